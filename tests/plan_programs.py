"""Programs that the re-planner takes, beside the ones that are timed (perf/cases.py), whose assembler they share."""
from __future__ import annotations

import perf.cases as cases


def residual_norm(rows, cols, dtype, lanes=148):
    """LayerNorm(x + y) gamma + beta: the norm of a post-norm transformer layer."""
    p = cases._Assembler(lanes)
    x, y = p.input((rows, cols), dtype), p.input((rows, cols), dtype)
    gamma, beta = p.input((cols,), dtype), p.input((cols,), dtype)
    out = p.chain((cases._ADD, (x, y), dtype))
    p.phase()
    out = p.rows(cases._LAYERNORM, out, rows, cols, cases._bits(1e-5))
    p.phase()
    by_col = p.view((rows, cols), (0, 1))
    out = p.chain((cases._MUL, (out, gamma), dtype, 0, by_col), (cases._ADD, (-1, beta), dtype, 0, by_col))
    p.output(out, (rows, cols))
    return p


def viewed_product(M, K, N, dtype, dims, strides, off, elems):
    """a @ w, where a is read from a buffer of `elems` elements through a view."""
    p = cases._Assembler(148)
    a, w = p.input((elems,), dtype), p.input((K, N), dtype)
    out = p.matmul(a, w, M, N, K, dtype, va=p.view(dims, strides, off))
    p.output(out, (M, N))
    return p


def products(dtype, *mkn):
    """Products that need nothing of each other, one phase."""
    p = cases._Assembler(148)
    for M, K, N in mkn:
        p.output(p.matmul(p.input((M, K), dtype), p.input((K, N), dtype), M, N, K, dtype), (M, N))
    return p


# a of 16 x 64 out of 1024 elements, as (2, 8, 64): blocks of eight rows, each block's rows last to first / first to last
REVERSED = (16, 64, 24, "f32", (2, 8, 64), (512, -64, 1), 448, 1024)
BLOCKED = (16, 64, 24, "f32", (8, 2, 64), (64, 512, 1), 0, 1024)


def widened_product(M, K, N, dtype, what):
    """A 16-bit product whose last value is converted to f32: of the product itself, or of what follows it in 16 bits."""
    p = cases._Assembler(148)
    a, w, x = p.input((M, K), dtype), p.input((K, N), dtype), p.input((M, N), dtype)
    y = p.matmul(a, w, M, N, K, dtype)
    p.phase()
    if what == "residual":
        y = p.chain((cases._ADD, (x, y), dtype))
    elif what == "gelu":
        y = p.chain((cases._GELU, (y,), dtype))
    elif what == "both":
        y = p.chain((cases._ADD, (x, y), dtype), (cases._GELU, (-1,), dtype))
    if what != "product":
        p.phase()
    p.output(p.chain((cases._CONVERT, (y,), "f32")), (M, N))
    return p


def product_then(M, K, N, dtype, what, transposed=False):
    """A 16-bit product and what follows it in its own type: nothing, a residual, a product with x ("times"), GELU (with the product
    kept: "kept"), a residual with the product kept ("both"); the f32 sum with an f32 x ("wide"); or as in a training step: times GELU's derivative at x ("grad"), x less a thousandth of it ("step"), its difference to x scaled, and the sum
    of the difference's squares ("loss")."""
    p = cases._Assembler(148)
    a, w, x = p.input((M, K), dtype), p.input((N, K) if transposed else (K, N), dtype), p.input((M, N), "f32" if what == "wide" else dtype)
    y = p.matmul(a, w, M, N, K, "f32" if what == "step" else dtype, vb=p.view((K, N), (1, K)) if transposed else 0)
    if what in ("kept", "both"):
        p.output(y, (M, N))
    if what in ("grad", "step"):
        xf = p.chain((cases._CONVERT, (x,), "f32"))
    if what != "product":
        p.phase()
    if what in ("residual", "both"):
        y = p.chain((cases._ADD, (x, y), dtype))
    elif what == "times":
        y = p.chain((cases._MUL, (y, x), dtype))
    elif what == "wide":
        y = p.chain((cases._CONVERT, (y,), "f32"), (cases._ADD, (-1, x), "f32"))
    elif what in ("gelu", "kept"):
        y = p.chain((cases._GELU, (y,), dtype))
    elif what == "grad":
        g, yf = p.region((xf,), M * N, cases._GELU_GRAD), p.chain((cases._CONVERT, (y,), "f32"))
        p.phase()
        y = p.chain((cases._MUL, (g, yf), "f32"), (cases._CONVERT, (-1,), dtype))
    elif what == "step":
        u = p.region((y, xf), M * N, ((cases._AFFINE, 2, 0, 0, 1e-3, 0.0), (cases._SUB, 0, 1, 2)))
        p.phase()
        y = p.chain((cases._CONVERT, (u,), dtype))
    elif what == "loss":
        yf, xf, diff = (p.buf(M * N, "f32") for _ in range(3))
        sq = p.chain((cases._CONVERT, (y,), yf), (cases._CONVERT, (x,), xf), (cases._SUB, (yf, xf), diff), (cases._MUL, (-1, -1), "f32"))
        p.phase()
        total = p.full_sum(sq)
        p.phase()
        y = p.chain((cases._AFFINE, (diff,), "f32", cases._bits(2.0 / (M * N)), 0), (cases._CONVERT, (-1,), dtype))
        p.output(total, ())
    p.output(y, (M, N))
    return p


def attention_of_sums(H, T, C, hd, dtype, causal, trips=0, by_key=False):
    """(q + q0) K^T, softmax, V: a program with an attention task that something around it lets the re-planner take. `trips`: the
    attention is the body of a loop; `by_key`: K as [H, C, hd], seen through its transpose."""
    p = cases._Assembler(148)
    q, q0 = p.input((H, T, hd), dtype), p.input((H, T, hd), dtype)
    k, v = p.input((H, C, hd) if by_key else (H, hd, C), dtype), p.input((H, C, hd), dtype)
    s = p.chain((cases._ADD, (q, q0), dtype))
    p.phase()
    if trips:
        p.loop = (len(p.phases) - 1, trips)
    p.output(p.attention(s, k, v, H, T, C, hd, causal, 0, p.view((H, hd, C), (C * hd, 1, hd)) if by_key else 0), (H, T, hd))
    return p


def stages(rows, cols, dtype, what, total=False):
    """x (+ y) (x gamma) (+ beta) (GELU), each as a task that rounds to `dtype`, and the sum of the result."""
    p = cases._Assembler(148)
    x = p.input((rows, cols), dtype)
    ops, by_col, cur = [], p.view((rows, cols), (0, 1)), x
    for w in what:
        if w == "res":
            ops.append((cases._ADD, (cur, p.input((rows, cols), dtype)), dtype))
        elif w == "gelu":
            ops.append((cases._GELU, (cur,), dtype))
        else:
            ops.append(({"mul": cases._MUL, "add": cases._ADD}[w], (cur, p.input((cols,), dtype)), dtype, 0, by_col))
        cur = -1
    out = x
    if ops:
        out = p.chain(*ops)
        p.output(out, (rows, cols))
        p.phase()
    if total:
        if dtype != "f32":
            out = p.chain((cases._CONVERT, (out,), "f32"))
            p.phase()
        p.output(p.full_sum(out), ())
    return p


def flat(n, dtype, ops):
    """A chain of elementwise ops over n elements (subops of perf/cases.py; the binary ones take a second argument each)."""
    p = cases._Assembler(148)
    cur, chain = p.input((n,), dtype), []
    for k in ops:
        chain.append((k, (cur,) if k in (cases._GELU, cases._TANH) else (cur, p.input((n,), dtype)), dtype))
        cur = -1
    p.output(p.chain(*chain), (n,))
    return p


def rms_norm(p, x, gain, rows, cols, dtype, eps):
    """x rsqrt(mean of squares + eps) gain, in the tile ops that a decoder block's norm arrives in."""
    half = dtype != "f32"
    xf = p.buf(rows * cols, "f32") if half else x
    p_sq = p.chain(*([(cases._CONVERT, (x,), xf)] if half else []), (cases._MUL, (xf, xf), "f32"))
    p.phase()
    ss = p.row_sums(p_sq, rows, cols)
    p.phase()
    r = p.region((ss,), rows, ((cases._AFFINE, 1, 0, 0, 1.0 / cols, eps), (cases._RSQRT, 0, 1, 1)))
    p.phase()
    by_row, by_col = p.view((rows, cols), (1, 0)), p.view((rows, cols), (0, 1))
    if not half:
        return p.chain((cases._MUL, (xf, r), "f32", 0, by_row), (cases._MUL, (-1, gain), "f32", 0, by_col))
    t = p.chain((cases._MUL, (xf, r), "f32", 0, by_row))
    gf = p.chain((cases._CONVERT, (gain,), "f32"))
    p.phase()
    return p.chain((cases._MUL, (t, gf), "f32", 0, by_col), (cases._CONVERT, (-1,), dtype))


def lone_norm(rows, cols, dtype, softmax):
    p = cases._Assembler(148)
    x = p.input((rows, cols), dtype)
    p.output(p.rows(cases._SOFTMAX, x, rows, cols) if softmax else p.rows(cases._LAYERNORM, x, rows, cols, cases._bits(1e-5)), (rows, cols))
    return p


def accelerations(p, at, mass, n):
    """sum_j m_j (|x_j - x_i|^2 + eps)^-1.5 (x_j - x_i), as a body of perf/cases.py's N-body loop."""
    d = p.buf(3 * n * n, "f32")
    sq = p.chain((cases._SUB, (at, at), d, p.view((n, n, 3), (0, 3, 1)), p.view((n, n, 3), (3, 0, 1))), (cases._MUL, (-1, -1), "f32"))
    p.phase()
    r2 = p.row_sums(sq, n * n, 3)
    p.phase()
    w = p.chain((cases._AFFINE, (r2,), "f32", cases._bits(1.0), cases._bits(1e-4)),
                (cases._POW, (-1, p.scalar(-1.5)), "f32", 0, p.view((n, n), (0, 0))), (cases._MUL, (-1, mass), "f32", 0, p.view((n, n), (0, 1))))
    p.phase()
    f = p.chain((cases._MUL, (d, w), "f32", 0, p.view((n, n, 3), (n, 1, 0))))
    p.phase()
    return p.strided_sum(f, 3 * n, n, 3)


def evaluations(n, steps, after=0):
    """Accelerations at x + s v for every s (0: at x itself), none of which needs another's. `after`: that many ops on the first
    one, plus x and then its sign turned, and what they make are the positions of one more."""
    p = cases._Assembler(148)
    x, v, mass = p.input((n, 3), "f32"), p.input((n, 3), "f32"), p.input((n,), "f32")
    at = [p.chain((cases._AFFINE, (v,), "f32", cases._bits(s), 0), (cases._ADD, (x, -1), "f32")) if s else x for s in steps]
    if any(steps):
        p.phase()
    outs = []
    for k, a in enumerate(at):
        if k:
            p.phase()
        outs.append(accelerations(p, a, mass, n))
    if after:
        p.phase()
        outs.append(p.chain((cases._ADD, (outs[0], x), "f32"), *[(cases._AFFINE, (-1,), "f32", cases._bits(-1.0), 0)] * (after - 1)))
        p.phase()
        outs.append(accelerations(p, outs[-1], mass, n))
    for a in outs:
        p.output(a, (n, 3))
    return p
