"""Programs that the re-planner takes, beside the ones that are timed (perf/cases.py), whose assembler they share."""
from __future__ import annotations

import perf.cases as cases


def residual_norm(rows, cols, dtype):
    """LayerNorm(x + y) gamma + beta: the norm of a post-norm transformer layer."""
    p = cases._Assembler(148)
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
