"""The work a user of this backend has it do, as cases to be timed.

A case is one VMProgram (the five benchmark configurations, at their own sizes and at others a
program of the same kind has), loaded once and executed through the package's public calls:
`VmProgram.Parse`, `LoadedProgram.Load`, then one `ExecuteDeviceAsync` per pass on buffers that
stay on the GPU, or one `Execute` on host arrays.

The programs are assembled here (the reference's lowering, which produced the committed blobs, is
not needed): the same tile ops, operand views, phases and lane shares as the committed programs of
the same kind have, at any size.
"""
import importlib
import math
import struct

import numpy as np
import torch

_PKG = "pjrt-ocl_b200"

# ---------------------------------------------------------------------------------------------
# the bytecode: dtypes, tile ops, elementwise subops
# ---------------------------------------------------------------------------------------------
_DT = {"f32": 0, "i32": 1, "f16": 6, "bf16": 7}
_SIZE = {"f32": 4, "i32": 4, "f16": 2, "bf16": 2}
_TORCH = {"f32": torch.float32, "i32": torch.int32, "f16": torch.float16, "bf16": torch.bfloat16}
_EW, _MMA, _GATHER, _RED_PART, _RED_COMB, _DYN_SCATTER = 0, 1, 2, 3, 4, 8
_RED_SEG, _SOFTMAX, _LAYERNORM, _REGION, _FLASH, _RED_STRIDED = 10, 11, 12, 13, 14, 15
_ADD, _MUL, _SUB, _MAX, _POW, _COPY, _RSQRT, _TANH = 0, 1, 2, 4, 6, 7, 12, 13
_CONVERT, _XOR, _AFFINE, _GELU = 23, 37, 40, 41
_BARRIER, _FOR, _NO_FLAG = 0xFFFFFFFE, 0xFFFFFFFB, 0xFFFFFFFF
_EW_TILE, _MMA_TILE = 4096, 128
# what one tile of a class costs a lane, as the scheduler that cut the committed programs was told
_COST = {_MMA: 20.0, _GATHER: 1.5}


def _bits(x):
    return struct.unpack("<I", struct.pack("<f", x))[0]


def _cdiv(a, b):
    return -(-a // b)


class _Assembler:
    """One straight-line program, with at most one counted loop at its end. `phase()` closes a
    phase; every call between two of them adds a unit of work (a task, or a chain of elementwise
    tasks over the same elements) to the open one."""

    def __init__(self, lanes):
        self.lanes = lanes
        self.bufs = []            # [elements, dtype, first phase, last phase, is argument / result / constant]
        self.dims = {}
        self.inputs, self.outputs = [], []
        self.consts, self.aux, self.tasks = [], [0], []
        self.phases = [[]]        # phase -> [(tasks, tiles, cost of a tile)]
        self.loop = None          # (index of its first phase, trips)

    # -- buffers ---------------------------------------------------------------------------
    def buf(self, n, dtype):
        self.bufs.append([n, dtype, None, 0, False])
        return len(self.bufs) - 1

    def input(self, shape, dtype):
        b = self.buf(math.prod(shape), dtype)
        self.bufs[b][4] = True
        self.dims[b] = tuple(shape)
        self.inputs.append(b)
        return b

    def scalar(self, value):
        b = self.buf(1, "f32")
        self.bufs[b][4] = True
        self.consts.append((b, struct.pack("<f", value)))
        return b

    def izero(self):
        b = self.buf(1, "i32")
        self.bufs[b][4] = True
        self.consts.append((b, struct.pack("<i", 0)))
        return b

    def output(self, b, shape):
        self.bufs[b][4] = True
        self.dims[b] = tuple(shape)
        self.outputs.append(b)

    def words(self, *w):
        self.aux += [int(x) & 0xFFFFFFFF for x in w]
        return len(self.aux) - len(w)

    def view(self, dims, strides, off=0):
        """An operand view; the value is what a task's view field holds."""
        return self.words(len(dims), *dims, *strides, off) + 1

    # -- tasks -------------------------------------------------------------------------------
    def _touch(self, *ids):
        ph = len(self.phases) - 1
        for b in ids:
            e = self.bufs[b]
            e[2] = ph if e[2] is None else min(e[2], ph)
            e[3] = max(e[3], ph)

    def _task(self, op, dst, a, b, *p, reads=(), adtype=None):
        dt = _DT[self.bufs[dst][1]]
        adt = _DT[self.bufs[a][1]] if adtype is None else _DT[adtype]
        self._touch(dst, a, b, *reads)
        self.tasks.append((op | dt << 8 | adt << 16, dst, a, b) + tuple(p) + (0,) * (8 - len(p)))
        return len(self.tasks) - 1

    def _unit(self, tasks, tiles, cost):
        self.phases[-1].append((tasks, tiles, cost))

    def phase(self):
        self.phases.append([])

    def chain(self, *ops):
        """Elementwise ops over the same elements, run by a lane one after another. An op is
        (subop, operands, result dtype[, p2, p3]); an operand -1 is the previous result."""
        prev, tasks, n = None, [], None
        for sub, operands, dtype, *p in ops:
            ids = [prev if x == -1 else x for x in operands]
            dst = None
            if isinstance(dtype, int):        # into this buffer
                dst = dtype
            a, b = ids[0], ids[-1]
            if dst is None:
                n_el = p[2] if len(p) > 2 else self.bufs[a][0]
                dst = self.buf(n_el, dtype)
            n = self.bufs[dst][0]
            tasks.append(self._task(_EW, dst, a, b, sub, n, *(p[:2] if p else (0, 0))))
            prev = dst
        self._unit(tasks, _cdiv(n, _EW_TILE), 1.0)
        return prev

    def matmul(self, a, b, M, N, K, dtype, va=0, vb=0, epilogue=None, residual=None):
        d = self.buf(M * N, dtype)
        e = r = 0
        if epilogue is not None:              # (micro-op, operand source): 1 = the residual
            e = self.words(1, epilogue[0], epilogue[1], 0, 0) + 1
            r = residual if residual is not None else 0
        t = self._task(_MMA, d, a, b, M, N, K, 1, va, vb, e, r, reads=() if residual is None else (residual,))
        self._unit([t], _cdiv(M, _MMA_TILE) * _cdiv(N, _MMA_TILE), _COST[_MMA])
        return d

    def rows(self, op, x, rows, seg, *p):
        d = self.buf(rows * seg, self.bufs[x][1])
        self._unit([self._task(op, d, x, 0, rows, seg, *p)], rows, 1.0)
        return d

    def row_sums(self, x, rows, seg):
        d = self.buf(rows, "f32")
        self._unit([self._task(_RED_SEG, d, x, 0, rows, seg, 0)], rows, 1.0)
        return d

    def full_sum(self, x):
        """Two phases: partial sums, then their sum."""
        n = self.bufs[x][0]
        chunk = _cdiv(_cdiv(n, 256), _EW_TILE) * _EW_TILE
        parts = _cdiv(n, chunk)
        part, out = self.buf(parts, "f32"), self.buf(1, "f32")
        self._unit([self._task(_RED_PART, part, x, 0, n, chunk, 0)], parts, chunk / _EW_TILE)
        self.phase()
        self._unit([self._task(_RED_COMB, out, part, 0, parts, 0)], 1, 1.0)
        return out

    def strided_sum(self, x, n_out, red, inner):
        d = self.buf(n_out, "f32")
        self._unit([self._task(_RED_STRIDED, d, x, 0, n_out, red, inner, 0)], _cdiv(n_out, _EW_TILE), 1.0)
        return d

    def region(self, ins, n, micro):
        """A fused elementwise program: micro-ops (subop, result slot, slot a, slot b[, s, t])."""
        d = self.buf(n, "f32")
        w = [len(ins), 0, len(micro)] + list(range(len(ins)))
        for k, dst, a, b, *st in micro:
            w += [k, dst, a, b] + [_bits(x) for x in st] + [0] * (2 - len(st))
        ids = list(ins) + [ins[0]] * (8 - len(ins))
        t = self._task(_REGION, d, ids[0], ids[1], self.words(*w), n, *ids[2:], reads=ids)
        self._unit([t], _cdiv(n, _EW_TILE), 1.0)
        return d

    def gather(self, x, n, dims, strides, off=0):
        d = self.buf(n, self.bufs[x][1])
        t = self._task(_GATHER, d, x, 0, self.words(len(dims), *dims, *strides, off), n)
        self._unit([t], _cdiv(n, _EW_TILE), _COST[_GATHER])
        return d

    def write_at(self, x, upd, dims, strides, clamp, starts):
        """Writes `upd` into `x` at run-time start indices."""
        r = len(dims)
        n = self.bufs[upd][0]
        w = self.words(r, *dims, *strides, *clamp, *([0] * r), *starts, 0)
        t = self._task(_DYN_SCATTER, x, upd, upd, w, n, reads=starts)
        self._unit([t], _cdiv(n, _EW_TILE), 1.0)

    def attention(self, q, k, v, H, T, C, hd, causal, vq=0, vk=0, vv=0):
        d = self.buf(H * T * hd, self.bufs[q][1])
        w = self.words(H, T, C, hd, _bits(1.0 / math.sqrt(hd)), 1 if causal else 0, vq, vk, vv)
        t = self._task(_FLASH, d, q, k, v, H, T, w, reads=(v,))
        self._unit([t], H * T, 1.0)
        return d

    # -- schedule and bytes -----------------------------------------------------------------------
    def _streams(self):
        """Entries of every lane. A unit gets a share of the lanes by its cost; its tiles are cut
        evenly into that many pieces and the pieces go to the least loaded lanes, largest first."""
        lanes = [[] for _ in range(self.lanes)]
        body_at = [0] * self.lanes
        root_len = [None] * self.lanes

        def put(lane, task, lo=0, hi=0, wait=_NO_FLAG, count=0):
            lanes[lane].append((task, lo, hi, wait, count, _NO_FLAG, 0, 0))

        for k, units in enumerate(self.phases):
            if self.loop and k == self.loop[0]:
                for l in range(self.lanes):
                    put(l, _BARRIER)
                    put(l, _FOR, len(lanes[l]) + 1, 0, self.loop[1])
                    root_len[l] = body_at[l] = len(lanes[l])
            elif k:
                for l in range(self.lanes):
                    put(l, _BARRIER)
            total = sum(t * c for _, t, c in units)
            pieces = []
            for tasks, tiles, cost in units:
                parts = max(1, min(tiles, math.ceil(self.lanes * tiles * cost / total)))
                for i in range(parts):
                    lo, hi = i * tiles // parts, (i + 1) * tiles // parts
                    pieces.append(((hi - lo) * cost, tasks, lo, hi))
            pieces.sort(key=lambda x: -x[0])
            load = [0.0] * self.lanes
            free = list(range(self.lanes))
            for w, tasks, lo, hi in pieces:
                l = free.pop(0) if free else min(range(self.lanes), key=load.__getitem__)
                load[l] += w
                for t in tasks:
                    put(l, t, lo, hi)
        if self.loop:
            for l in range(self.lanes):
                e = lanes[l][body_at[l] - 1]
                lanes[l][body_at[l] - 1] = (e[0], e[1], len(lanes[l]) - body_at[l]) + e[3:]
        return lanes, root_len

    def _place(self):
        """Byte offsets in the arena: buffers whose phases do not overlap share memory, except
        arguments, results, constants and whatever lives in the loop."""
        offs, end, live = [0] * len(self.bufs), 0, []
        own = [b for b in range(len(self.bufs)) if self.bufs[b][4] or
               (self.loop and self.bufs[b][3] >= self.loop[0])]
        kept = set(own)
        rest = sorted((b for b in range(len(self.bufs)) if b not in kept), key=lambda b: self.bufs[b][2] or 0)
        size = lambda b: (self.bufs[b][0] * _SIZE[self.bufs[b][1]] + 63) // 64 * 64   # noqa: E731
        for b in rest:
            first = self.bufs[b][2] or 0
            live = [x for x in live if self.bufs[x][3] >= first]
            at = 0
            for x in sorted(live, key=lambda x: offs[x]):
                if at + size(b) <= offs[x]:
                    break
                at = max(at, offs[x] + size(x))
            offs[b] = at
            live.append(b)
            end = max(end, at + size(b))
        for b in own:
            offs[b] = end
            end += size(b)
        return offs, end

    def blob(self):
        offs, arena = self._place()
        lanes, root_len = self._streams()
        out = bytearray()

        def pad():
            out.extend(b"\0" * (-len(out) % 8))
        out += struct.pack("<IIIIIIIIIIQ", 0x314D5056, 3, len(self.bufs), 0, len(self.consts), 0,
                           len(self.inputs), len(self.outputs), len(self.aux), 0, arena)
        for (n, dt, *_), off in zip(self.bufs, offs):
            out += struct.pack("<QQII", off, n * _SIZE[dt], _DT[dt], 0)
        for ids in (self.inputs, self.outputs):
            out += struct.pack("<%dI" % len(ids), *ids)
            pad()
        for b in self.inputs + self.outputs:
            out += struct.pack("<II%dQ" % len(self.dims[b]), len(self.dims[b]), 0, *self.dims[b])
        out += struct.pack("<%dI" % len(self.aux), *self.aux)
        pad()
        for b, data in self.consts:
            out += struct.pack("<II", b, len(data)) + data
            pad()
        out += struct.pack("<IIII", len(self.tasks), sum(map(len, lanes)), 0, len(lanes))
        for t in self.tasks:
            out += struct.pack("<12I", *t)
        at = 0
        for l, stream in enumerate(lanes):
            out += struct.pack("<IIII", at, len(stream), root_len[l] or len(stream), 0)
            at += len(stream)
        for stream in lanes:
            for e in stream:
                out += struct.pack("<8I", *e)
        return bytes(out)


# ---------------------------------------------------------------------------------------------
# programs
# ---------------------------------------------------------------------------------------------
def _relu_matmul(c):
    """maximum(a @ w, 0)."""
    M, K, N, dt = c["m"], c["k"], c["n"], c["dtype"]
    p = _Assembler(148)
    a, w = p.input((M, K), dt), p.input((K, N), dt)
    y = p.matmul(a, w, M, N, K, dt)
    p.phase()
    out = p.chain((_MAX, (y, p.scalar(0.0)), "f32", 0, p.view((M, N), (0, 0))))
    p.output(out, (M, N))
    return p


def _dot(c):
    """a @ w, or a @ w^T with both operands contiguous along k."""
    M, K, N, dt = c["m"], c["k"], c["n"], c["dtype"]
    p = _Assembler(148)
    a = p.input((M, K), dt)
    w = p.input((N, K) if c["transposed"] else (K, N), dt)
    out = p.matmul(a, w, M, N, K, dt, vb=p.view((K, N), (1, K)) if c["transposed"] else 0)
    p.output(out, (M, N))
    return p


def _norm_chain(c):
    """LayerNorm, times gamma plus beta, tanh-GELU, softmax, and the sum of everything."""
    R, C, dt = c["rows"], c["cols"], c["dtype"]
    p = _Assembler(148)
    x, gamma, beta = p.input((R, C), dt), p.input((C,), dt), p.input((C,), dt)
    core = p.rows(_LAYERNORM, x, R, C, _bits(1e-5))
    p.phase()
    y = p.chain((_MUL, (core, gamma), dt, 0, p.view((R, C), (0, 1))),
                (_ADD, (-1, beta), dt, 0, p.view((R, C), (0, 1))), (_GELU, (-1,), dt))
    p.phase()
    sm = p.rows(_SOFTMAX, y, R, C)
    p.phase()
    s = sm
    if dt != "f32":
        s = p.chain((_CONVERT, (sm,), "f32"))
        p.phase()
    total = p.full_sum(s)
    p.output(sm, (R, C))
    p.output(total, ())
    return p


def _int_chain(c):
    """maximum((a + b) ^ c, d)."""
    R, C = c["rows"], c["cols"]
    p = _Assembler(148)
    a, b, x, y = (p.input((R, C), "i32") for _ in range(4))
    out = p.chain((_ADD, (a, b), "i32"), (_XOR, (-1, x), "i32"), (_MAX, (-1, y), "i32"))
    p.output(out, (R, C))
    return p


# d/dz of tanh-GELU, as the reference's region pass leaves it (slot 0 is z, and the result)
_K0, _K1 = 0.7978845608, 0.044715
_GELU_GRAD = ((_MUL, 1, 0, 0), (_MUL, 2, 1, 0), (_AFFINE, 3, 2, 2, _K1, 0.0), (_ADD, 2, 0, 3),
              (_AFFINE, 3, 2, 2, _K0, 0.0), (_TANH, 2, 3, 3), (_MUL, 3, 2, 2), (_AFFINE, 4, 3, 3, -1.0, 1.0),
              (_AFFINE, 3, 1, 1, 3 * _K0 * _K1, _K0), (_AFFINE, 1, 2, 2, 0.5, 0.5), (_AFFINE, 2, 0, 0, 0.5, 0.0),
              (_MUL, 0, 4, 3), (_MUL, 3, 2, 0), (_ADD, 0, 1, 3))
_LR = 1e-3


def _mlp(c):
    """Three layers forward, mean squared error, the gradients and one SGD step."""
    B, d0, d1, d2, d3, dt = c["batch"], c["d0"], c["d1"], c["d2"], c["d3"], c["dtype"]
    half = dt != "f32"
    p = _Assembler(144)
    x, y = p.input((B, d0), dt), p.input((B, d3), dt)
    ws = [p.input(s, dt) for s in ((d0, d1), (d1, d2), (d2, d3))]
    w1, w2, w3 = ws

    def tr(r, k):                 # the transpose of a [k, r] buffer
        return p.view((r, k), (1, r))
    z1 = p.matmul(x, w1, B, d1, d0, dt)
    p.phase()
    h1 = p.chain((_GELU, (z1,), dt))
    p.phase()
    z2 = p.matmul(h1, w2, B, d2, d1, dt)
    p.phase()
    h2 = p.chain((_GELU, (z2,), dt))
    p.phase()
    pr = p.matmul(h2, w3, B, d3, d2, dt)
    p.phase()
    n3 = B * d3
    scale = (_AFFINE, None, "f32", _bits(2.0 / n3), 0)
    if half:
        pf, yf, diff = (p.buf(n3, "f32") for _ in range(3))
        sq = p.chain((_CONVERT, (pr,), pf), (_CONVERT, (y,), yf), (_SUB, (pf, yf), diff), (_MUL, (-1, -1), "f32"))
    else:
        diff = p.buf(n3, "f32")
        sq = p.chain((_SUB, (pr, y), diff), (_MUL, (-1, -1), "f32"))
    p.phase()
    total = p.full_sum(sq)
    p.phase()
    loss = p.chain((_MUL, (total, p.scalar(1.0 / n3)), "f32"))
    scaled = (scale[0], (diff,)) + scale[2:]
    dp = p.chain(scaled, (_CONVERT, (-1,), dt)) if half else p.chain(scaled)
    p.phase()
    dw3 = p.matmul(h2, dp, d2, d3, B, "f32", va=tr(d2, B))
    dh2 = p.matmul(dp, w3, B, d2, d3, dt, vb=p.view((d3, d2), (1, d3)))
    z2f = p.chain((_CONVERT, (z2,), "f32")) if half else z2
    p.phase()

    def backward(z_f32, dh, n):
        g = p.region((z_f32,), n, _GELU_GRAD)
        if half:
            dhf = p.chain((_CONVERT, (dh,), "f32"))
            p.phase()
            dz = p.chain((_MUL, (g, dhf), "f32"), (_CONVERT, (-1,), dt))
        else:
            p.phase()
            dz = p.chain((_MUL, (g, dh), "f32"))
        p.phase()
        return dz
    dz2 = backward(z2f, dh2, B * d2)
    dw2 = p.matmul(h1, dz2, d1, d2, B, "f32", va=tr(d1, B))
    dh1 = p.matmul(dz2, w2, B, d1, d2, dt, vb=p.view((d2, d1), (1, d2)))
    z1f = p.chain((_CONVERT, (z1,), "f32")) if half else z1
    p.phase()
    dz1 = backward(z1f, dh1, B * d1)
    dw1 = p.matmul(x, dz1, d0, d1, B, "f32", va=tr(d0, B))
    step = ((_AFFINE, 2, 0, 0, _LR, 0.0), (_SUB, 0, 1, 2))
    new = []
    if half:
        wf = [p.chain((_CONVERT, (w1,), "f32")), None, None]
        p.phase()
        sizes = (d0 * d1, d1 * d2, d2 * d3)
        for i, dw in enumerate((dw1, dw2, dw3)):
            u = p.region((dw, wf[i]), sizes[i], step)
            p.phase()
            new.append(p.chain((_CONVERT, (u,), dt)))
            if i < 2:
                wf[i + 1] = p.chain((_CONVERT, (ws[i + 1],), "f32"))
                p.phase()
    else:
        p.phase()
        for w, dw, n in ((w1, dw1, d0 * d1), (w2, dw2, d1 * d2), (w3, dw3, d2 * d3)):
            new.append(p.region((dw, w), n, step))
    p.output(loss, ())
    for b, s in zip(new, ((d0, d1), (d1, d2), (d2, d3))):
        p.output(b, s)
    return p


def _rms_norm(p, x, gain, n, d, dt, chained=None):
    """RMS norm of n rows of d, decomposed. `chained`: elementwise ops that make `x` in the first
    phase (the residual sum). Returns (x, the normalised rows)."""
    half = dt != "f32"
    ops = []
    if chained is not None:
        x = p.buf(n * d, dt)
        ops.append(chained + (x,))
    if half:
        xf = p.buf(n * d, "f32")
        ops += [(_CONVERT, (x,), xf)]
    else:
        xf = x
    sq = p.chain(*ops, (_MUL, (xf, xf), "f32"))
    p.phase()
    ss = p.row_sums(sq, n, d)
    p.phase()
    r = p.region((ss,), n, ((_AFFINE, 1, 0, 0, 1.0 / d, 1e-6), (_RSQRT, 0, 1, 1)))
    p.phase()
    by_row = p.view((n, d), (1, 0))
    by_col = p.view((n, d), (0, 1))
    if half:
        t = p.chain((_MUL, (xf, r), "f32", 0, by_row))
        gf = p.chain((_CONVERT, (gain,), "f32"))
        p.phase()
        h = p.chain((_MUL, (t, gf), "f32", 0, by_col), (_CONVERT, (-1,), dt))
    else:
        h = p.chain((_MUL, (xf, r), "f32", 0, by_row), (_MUL, (-1, gain), "f32", 0, by_col))
    p.phase()
    return x, h


def _feed_forward(p, x1, h2, w1, w2, n, d, f, dt):
    up = p.matmul(h2, w1, n, f, d, dt, epilogue=(_GELU, 0))
    p.phase()
    if dt == "f32":               # the residual sum is the matmul's store epilogue
        return p.matmul(up, w2, n, d, f, dt, epilogue=(_ADD, 1), residual=x1)
    down = p.matmul(up, w2, n, d, f, dt)
    p.phase()
    return p.chain((_ADD, (x1, down), dt))


def _block(c):
    """Pre-norm decoder block forward (prefill): causal attention over heads of 64, GELU FFN."""
    b, s, H, dt = c["batch"], c["seq"], c["heads"], c["dtype"]
    hd, d, f, n = 64, c["heads"] * 64, c["heads"] * 256, c["batch"] * c["seq"]
    p = _Assembler(144)
    g1 = p.input((d,), dt)
    x = p.input((n, d), dt)
    wq, wk, wv, wo = (p.input((d, d), dt) for _ in range(4))
    g2 = p.input((d,), dt)
    w1, w2 = p.input((d, f), dt), p.input((f, d), dt)
    _, h = _rms_norm(p, x, g1, n, d, dt)
    q, k, v = (p.matmul(h, w, n, d, d, dt) for w in (wq, wk, wv))
    p.phase()
    heads = p.view((b, H, s, hd), (s * d, hd, d, 1))
    keys = p.view((b, H, hd, s), (s * d, hd, 1, d))
    o = p.attention(q, k, v, b * H, s, s, hd, True, heads, keys, p.view((b, H, s, hd), (s * d, hd, d, 1)))
    p.phase()
    merge = ((b, s, H, hd), (H * s * hd, hd, s * hd, 1))
    if dt == "f32":               # the merge of the heads is an operand view
        x1 = p.matmul(o, wo, n, d, d, dt, va=p.view(*merge), epilogue=(_ADD, 1), residual=x)
        p.phase()
        x1, h2 = _rms_norm(p, x1, g2, n, d, dt)
    else:
        o2 = p.gather(o, n * d, *merge)
        p.phase()
        attn = p.matmul(o2, wo, n, d, d, dt)
        p.phase()
        x1, h2 = _rms_norm(p, None, g2, n, d, dt, chained=(_ADD, (x, attn)))
    p.output(_feed_forward(p, x1, h2, w1, w2, n, d, f, dt), (n, d))
    return p


def _decode(c):
    """One decode step: one new token per sequence against caches that are updated in place."""
    b, cache, H, dt = c["batch"], c["cache"], c["heads"], c["dtype"]
    hd, d, f, C = 64, c["heads"] * 64, c["heads"] * 256, c["cache"] + 1
    p = _Assembler(144)
    g1 = p.input((d,), dt)
    x = p.input((b, d), dt)
    kc, vc = p.input((b * H, C, hd), dt), p.input((b * H, C, hd), dt)
    pos = p.input((), "i32")
    wq, wk, wv, wo = (p.input((d, d), dt) for _ in range(4))
    g2 = p.input((d,), dt)
    w1, w2 = p.input((d, f), dt), p.input((f, d), dt)
    zero = p.izero()
    _, h = _rms_norm(p, x, g1, b, d, dt)
    q, k, v = (p.matmul(h, w, b, d, d, dt) for w in (wq, wk, wv))
    p.phase()
    for buf, new in ((kc, k), (vc, v)):
        p.write_at(buf, new, (b * H, 1, hd), (C * hd, hd, 1), (0, cache, 0), (zero, pos, zero))
    p.phase()
    o = p.attention(q, kc, vc, b * H, 1, C, hd, True, 0, p.view((b * H, hd, C), (C * hd, 1, hd)))
    p.phase()
    if dt == "f32":
        x1 = p.matmul(o, wo, b, d, d, dt, epilogue=(_ADD, 1), residual=x)
        p.phase()
        x1, h2 = _rms_norm(p, x1, g2, b, d, dt)
    else:
        attn = p.matmul(o, wo, b, d, d, dt)
        p.phase()
        x1, h2 = _rms_norm(p, None, g2, b, d, dt, chained=(_ADD, (x, attn)))
    p.output(_feed_forward(p, x1, h2, w1, w2, b, d, f, dt), (b, d))
    for buf in (kc, vc):
        p.output(buf, (b * H, C, hd))
    return p


def _nbody(c):
    """All-pairs gravity, RK4, in a counted loop."""
    n, dt, soft = c["bodies"], 1e-3, 1e-2
    p = _Assembler(148)
    pos0, vel0, mass = p.input((n, 3), "f32"), p.input((n, 3), "f32"), p.input((n,), "f32")
    pos, vel = p.buf(3 * n, "f32"), p.buf(3 * n, "f32")
    p.chain((_COPY, (pos0,), pos))
    p.chain((_COPY, (vel0,), vel))
    p.phase()
    p.loop = (len(p.phases) - 1, c["steps"])
    expo = p.scalar(-1.5)

    def accel(at, carried):
        pj, pi = ((n, n, 3), (0, 3, 1)), ((n, n, 3), (3, 0, 1))
        if carried:               # positions that the loop carries are read through gathers
            a, b = p.gather(at, 3 * n * n, *pj), p.gather(at, 3 * n * n, *pi)
            p.phase()
            diff = (_SUB, (a, b))
            views = ()
        else:
            diff, views = (_SUB, (at, at)), (p.view(*pj), p.view(*pi))
        d = p.buf(3 * n * n, "f32")
        sq = p.chain(diff + (d,) + views, (_MUL, (-1, -1), "f32"))
        p.phase()
        r2 = p.buf(n * n, "f32")
        t = p._task(_RED_SEG, r2, sq, 0, n * n, 3, 0)
        p._unit([t], n * n, 1.0)
        p.phase()
        w = p.chain((_AFFINE, (r2,), "f32", _bits(1.0), _bits(soft * soft)),
                    (_POW, (-1, expo), "f32", 0, p.view((n, n), (0, 0))),
                    (_MUL, (-1, mass), "f32", 0, p.view((n, n), (0, 1))))
        p.phase()
        f = p.chain((_MUL, (d, w), "f32", 0, p.view((n, n, 3), (n, 1, 0))))
        p.phase()
        return p.strided_sum(f, 3 * n, n, 3)

    def times(x, s):
        return (_AFFINE, (x,), "f32", _bits(s), 0)
    k1v = accel(pos, True)
    x2 = p.chain(times(vel, dt / 2), (_ADD, (pos, -1), "f32"))
    p.phase()
    k2v = accel(x2, False)
    k2x, k3x, k4x = (p.buf(3 * n, "f32") for _ in range(3))
    x3 = p.chain(times(k1v, dt / 2), (_ADD, (vel, -1), k2x), times(k2x, dt / 2), (_ADD, (pos, -1), "f32"))
    p.phase()
    k3v = accel(x3, False)
    x4 = p.chain(times(k2v, dt / 2), (_ADD, (vel, -1), k3x), times(k3x, dt), (_ADD, (pos, -1), "f32"))
    p.phase()
    k4v = accel(x4, False)
    a = p.buf(3 * n, "f32")
    sx = p.buf(3 * n, "f32")
    b = p.buf(3 * n, "f32")
    p.chain(times(k3v, dt), (_ADD, (vel, -1), k4x), times(k2x, 2.0), (_ADD, (vel, -1), a),
            times(k3x, 2.0), (_ADD, (-1, k4x), b), (_ADD, (a, b), sx))
    p.phase()
    u, v, sv = (p.buf(3 * n, "f32") for _ in range(3))
    p.chain(times(k2v, 2.0), (_ADD, (k1v, -1), u), times(k3v, 2.0), (_ADD, (-1, k4v), v), (_ADD, (u, v), sv))
    p.phase()
    p.chain(times(sx, dt / 6), (_ADD, (pos, -1), "f32"), (_COPY, (-1,), pos))
    p.chain(times(sv, dt / 6), (_ADD, (vel, -1), "f32"), (_COPY, (-1,), vel))
    p.output(pos, (n, 3))
    p.output(vel, (n, 3))
    return p


_BUILD = {"relu_matmul": _relu_matmul, "dot": _dot, "norm_chain": _norm_chain, "int_chain": _int_chain,
          "mlp": _mlp, "block": _block, "decode": _decode, "nbody": _nbody}


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: config 1, relu(a @ w). What it takes is launch and latency.
        {"name": "relu_matmul", "kind": "relu_matmul", "m": 256, "k": 128, "n": 64, "dtype": "f32", "call": "device"},
        # The same through the synchronous call on host arrays, as a first jit of a small function runs.
        {"name": "relu_matmul_host", "kind": "relu_matmul", "m": 256, "k": 128, "n": 64, "dtype": "f32", "call": "host"},
        # Config 2: the elementwise / row-norm / reduction chain, at its size in f32.
        {"name": "norm_chain_f32", "kind": "norm_chain", "rows": 8192, "cols": 4096, "dtype": "f32"},
        # The same kind of work on 16-bit storage with rows that are no power of two.
        {"name": "norm_chain_bf16_ragged", "kind": "norm_chain", "rows": 3001, "cols": 1000, "dtype": "bf16"},
        # Config 2's integer chain.
        {"name": "int_chain", "kind": "int_chain", "rows": 8192, "cols": 4096},
        # One dot_general on its own, the size that the matmul tile op is quoted at.
        {"name": "dot_bf16", "kind": "dot", "m": 4096, "k": 4096, "n": 4096, "dtype": "bf16", "transposed": False},
        # Config 3: a training step, forward and backward, of the three-layer MLP.
        {"name": "mlp_step_bf16", "kind": "mlp", "batch": 8192, "d0": 1024, "d1": 4096, "d2": 4096, "d3": 1024,
         "dtype": "bf16"},
        # Config 5: prefill of the decoder block, the headline.
        {"name": "block_bf16", "kind": "block", "batch": 8, "seq": 2048, "heads": 16, "dtype": "bf16"},
        # Prefill of prompts whose length divides nothing, a width of 768.
        {"name": "block_bf16_ragged", "kind": "block", "batch": 3, "seq": 777, "heads": 12, "dtype": "bf16"},
        # The block in f32, the default type of a jax program, at the reference's own "base" size.
        {"name": "block_f32", "kind": "block", "batch": 4, "seq": 128, "heads": 8, "dtype": "f32"},
        # Config 5: one decode step against full caches, updated in place.
        {"name": "decode_bf16", "kind": "decode", "batch": 32, "cache": 2048, "heads": 16, "dtype": "bf16"},
        # Config 4: the N-body loop at its 4096 bodies, ten of its RK4 steps.
        {"name": "nbody", "kind": "nbody", "bodies": 4096, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step, odd=0.4):
    """A size from lo to hi, even over its logarithm: any number, or a multiple of `step`."""
    v = _log(rng, lo, hi)
    return v if rng.random() < odd else min(hi, max(step, v // step * step))


def draw(rng):
    kind = rng.choice(["relu_matmul", "norm_chain", "norm_chain", "int_chain", "dot", "mlp", "mlp", "block", "block",
                       "decode", "decode", "nbody"])
    c = {"kind": kind}
    if kind == "relu_matmul":
        c.update(m=_log(rng, 16, 512), k=_log(rng, 16, 512), n=_log(rng, 16, 512), dtype="f32",
                 call=rng.choice(["device", "host"]))
    elif kind == "norm_chain":
        c.update(rows=_log(rng, 64, 8192), cols=_size(rng, 128, 4096, 128), dtype=rng.choice(["f32", "bf16", "bf16", "f16"]))
    elif kind == "int_chain":
        c.update(rows=_log(rng, 64, 8192), cols=_size(rng, 128, 4096, 128))
    elif kind == "dot":
        dt = rng.choice(["bf16", "bf16", "f16", "f32"])
        top = 1024 if dt == "f32" else 4096
        c.update(m=_size(rng, 128, top, 64), k=_size(rng, 128, top, 64, 0.2), n=_size(rng, 128, top, 64, 0.2), dtype=dt,
                 transposed=rng.random() < 0.5)
    elif kind == "mlp":
        dt = rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
        plain = dt != "f32" and rng.random() < 0.8      # widths that are whole 16-byte words
        top, most = (4096, 8192) if plain else (512, 2048)
        w = [_size(rng, 64, top, 64, 0.0) if plain else _log(rng, 64, top) for _ in range(4)]
        c.update(batch=_log(rng, 64, most) // 8 * 8 + (0 if plain and rng.random() < 0.7 else rng.randrange(8)),
                 d0=w[0], d1=w[1], d2=w[2], d3=w[3], dtype=dt)
        c["batch"] = min(c["batch"], 8192)
    elif kind == "block":
        dt = rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
        if dt == "f32":
            c.update(batch=rng.randint(1, 4), seq=_size(rng, 32, 256, 32), heads=rng.choice([4, 8]), dtype=dt)
        else:
            c.update(batch=rng.randint(1, 8), seq=_size(rng, 64, 2048, 64), heads=rng.choice([4, 8, 12, 16]), dtype=dt)
    elif kind == "decode":
        dt = rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
        top = 4 if dt == "f32" else 32
        c.update(batch=_log(rng, 1, top), cache=_log(rng, 64, 2048), heads=rng.choice([4, 8, 12, 16]), dtype=dt)
    else:
        c.update(bodies=_size(rng, 256, 4096, 64), steps=rng.randint(2, 10))
    return c


_STATE = {}


def _runtime():
    """What a process keeps once: the runtime and the stream that it launches on."""
    if not _STATE:
        vm = importlib.import_module(_PKG)
        _STATE.update(vm=vm, rt=vm.Runtime.Create(torch.cuda.current_device()), stream=torch.cuda.Stream())
    return _STATE


def _inputs(c, gen):
    """Arguments in order, with the distributions of the benchmark configurations."""
    dev = "cuda"

    def normal(shape, dtype, scale=1.0, shift=0.0):
        return (torch.randn(shape, generator=gen, device=dev) * scale + shift).to(_TORCH[dtype])

    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=gen, device=dev) * (hi - lo) + lo
    k, dt = c["kind"], c.get("dtype")
    if k == "relu_matmul":
        return [normal((c["m"], c["k"]), dt), normal((c["k"], c["n"]), dt)]
    if k == "dot":
        w = (c["n"], c["k"]) if c["transposed"] else (c["k"], c["n"])
        return [normal((c["m"], c["k"]), dt), normal(w, dt, 1.0 / math.sqrt(c["k"]))]
    if k == "norm_chain":
        return [normal((c["rows"], c["cols"]), dt), normal((c["cols"],), dt, 0.1, 1.0), normal((c["cols"],), dt, 0.1)]
    if k == "int_chain":
        return [torch.randint(-2**20, 2**20, (c["rows"], c["cols"]), generator=gen, device=dev, dtype=torch.int32)
                for _ in range(4)]
    if k == "mlp":
        d = (c["d0"], c["d1"], c["d2"], c["d3"])
        return ([normal((c["batch"], d[0]), dt), normal((c["batch"], d[3]), dt)] +
                [normal((i, o), dt, 1.0 / math.sqrt(i)) for i, o in zip(d, d[1:])])
    if k == "nbody":
        n = c["bodies"]
        return [uniform((n, 3), -1.0, 1.0), normal((n, 3), "f32", 0.1), uniform((n,), 0.5, 1.5)]
    d, f = c["heads"] * 64, c["heads"] * 256
    gain = normal((d,), dt, 0.1, 1.0)
    tail = ([normal((d, d), dt, 0.02) for _ in range(4)] +
            [normal((d,), dt, 0.1, 1.0), normal((d, f), dt, 0.02), normal((f, d), dt, 0.02)])
    if k == "block":
        return [gain, normal((c["batch"] * c["seq"], d), dt)] + tail
    caches = [normal((c["batch"] * c["heads"], c["cache"] + 1, 64), dt) for _ in range(2)]
    pos = torch.full((), c["cache"], device=dev, dtype=torch.int32)
    return [gain, normal((c["batch"], d), dt)] + caches + [pos] + tail


def prepare(case, seed):
    s = _runtime()
    vm = s["vm"]
    asm = _BUILD[case["kind"]](case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    args = _inputs(case, gen)
    lp = vm.LoadedProgram.Load(s["rt"], vm.VmProgram.Parse(asm.blob()))
    if case.get("call") == "host":
        return {"lp": lp, "host": [a.cpu().numpy() for a in args]}
    outs = [torch.empty(asm.dims[b], dtype=_TORCH[asm.bufs[b][1]], device="cuda") for b in asm.outputs]
    for i, o in lp.InOutResults().items():        # a cache that is updated in place is its own result
        outs[o] = args[i]
    torch.cuda.synchronize()                      # the arguments are made on another stream
    return {"lp": lp, "args": args, "outs": outs, "stream": s["stream"].cuda_stream,
            "in_ptr": [a.data_ptr() for a in args], "out_ptr": [o.data_ptr() for o in outs]}


def run(state):
    if "host" in state:
        return state["lp"].Execute(state["host"])
    state["lp"].ExecuteDeviceAsync(state["in_ptr"], state["out_ptr"], state["stream"])
    return state["outs"]


def work(case):
    c, k = case, case["kind"]
    e = _SIZE.get(c.get("dtype", "f32"), 4)
    if k == "relu_matmul" or k == "dot":
        m, n, q = c["m"], c["n"], c["k"]
        return {"bytes": e * (m * q + q * n + m * n), "flops": 2 * m * n * q}
    if k == "norm_chain":
        n = c["rows"] * c["cols"]
        return {"bytes": 2 * e * n + 2 * e * c["cols"] + 4, "flops": 30 * n}
    if k == "int_chain":
        n = c["rows"] * c["cols"]
        return {"bytes": 20 * n, "flops": 3 * n}
    if k == "mlp":
        b, d = c["batch"], (c["d0"], c["d1"], c["d2"], c["d3"])
        w = [i * o for i, o in zip(d, d[1:])]
        return {"bytes": e * (b * (d[0] + d[3]) + 2 * sum(w)) + 4, "flops": 2 * b * (3 * sum(w) - w[0])}
    if k == "nbody":
        n = c["bodies"]
        return {"bytes": 4 * 13 * n, "flops": 20 * n * n * 4 * c["steps"]}
    d, f, b = c["heads"] * 64, c["heads"] * 256, c["batch"]
    weights = 4 * d * d + 2 * d * f + 2 * d
    if k == "block":
        n, s = b * c["seq"], c["seq"]
        return {"bytes": e * (weights + 2 * n * d), "flops": 2 * n * (4 * d * d + 2 * d * f) + 2 * b * s * (s + 1) * d}
    kv = 2 * b * (c["cache"] + 1) * d
    return {"bytes": e * (weights + kv + 2 * b * d), "flops": 2 * b * (4 * d * d + 2 * d * f) + 2 * kv}


def tolerance(case):
    if case["kind"] == "int_chain":
        return "exact"
    return {"rel": 1e-5} if case.get("dtype", "f32") == "f32" else {"rel": 1e-2}
