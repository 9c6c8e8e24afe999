"""Re-planned programs against a float64 reference, at the sizes where their kernels' tiles, splits and remainders meet."""
from __future__ import annotations

import pytest

import plan_programs as progs

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _rms(x, g):
    return x * torch.rsqrt((x * x).mean(1, keepdim=True) + 1e-6) * g


def _reference(c, args):
    a = [x.double() if x.is_floating_point() else x for x in args]
    k, h = c["kind"], c.get("heads")
    sdpa = torch.nn.functional.scaled_dot_product_attention
    if k == "relu_matmul":
        return [(a[0] @ a[1]).clamp(min=0)]
    if k == "dot":
        return [a[0] @ (a[1].T if c["transposed"] else a[1])]
    if k == "norm_chain":
        y = (a[0] - a[0].mean(1, keepdim=True)) / torch.sqrt(a[0].var(1, unbiased=False, keepdim=True) + 1e-5)
        s = torch.softmax(_gelu(y * a[1] + a[2]), 1)
        return [s, s.sum()]
    if k == "int_chain":
        return [torch.maximum((a[0] + a[1]) ^ a[2], a[3])]
    if k == "mlp":
        ws = [w.clone().requires_grad_() for w in a[2:5]]
        loss = ((_gelu(_gelu(a[0] @ ws[0]) @ ws[1]) @ ws[2] - a[1]) ** 2).mean()
        loss.backward()
        return [loss.detach()] + [w.detach() - 1e-3 * w.grad for w in ws]
    if k == "block":
        g1, x, wq, wk, wv, wo, g2, w1, w2 = a
        b, s = c["batch"], c["seq"]
        y = _rms(x, g1)
        q, kk, v = ((y @ w).view(b, s, h, 64).transpose(1, 2) for w in (wq, wk, wv))
        x1 = x + sdpa(q, kk, v, is_causal=True).transpose(1, 2).reshape(x.shape) @ wo
        return [x1 + _gelu(_rms(x1, g2) @ w1) @ w2]
    if k == "decode":
        g1, x, kc, vc, _, wq, wk, wv, wo, g2, w1, w2 = a
        n = c["batch"] * h
        y, kc, vc = _rms(x, g1), kc.clone(), vc.clone()
        kc[:, -1], vc[:, -1] = (y @ wk).view(n, 64), (y @ wv).view(n, 64)
        x1 = x + sdpa((y @ wq).view(n, 1, 64), kc, vc).view(c["batch"], -1) @ wo
        return [x1 + _gelu(_rms(x1, g2) @ w1) @ w2, kc, vc]
    p, v, m = a
    dt = 1e-3

    def acc(p):
        d = p[None] - p[:, None]
        return (d * ((d * d).sum(2) + 1e-4).pow(-1.5).mul(m[None])[..., None]).sum(1)
    for _ in range(c["steps"]):
        a1 = acc(p); v2 = v + dt / 2 * a1
        a2 = acc(p + dt / 2 * v); v3 = v + dt / 2 * a2
        a3 = acc(p + dt / 2 * v2); v4 = v + dt * a3
        a4 = acc(p + dt * v3)
        p, v = p + dt / 6 * (v + 2 * v2 + 2 * v3 + v4), v + dt / 6 * (a1 + 2 * a2 + 2 * a3 + a4)
    return [p, v]


def _case(kind, **kw):
    return pytest.param(dict(kind=kind, **kw), id="-".join([kind, *(str(v) for v in kw.values())]))


@pytest.mark.parametrize("c", [
    # CUDA-core products: one tile, ragged edges, K of one block / not a multiple of a block, every tile shape
    *(_case("dot", m=m, k=k, n=n, dtype="f32", transposed=t) for m, k, n, t in
      [(1, 1, 1, False), (17, 33, 15, True), (130, 100, 66, False), (512, 16, 384, True), (700, 250, 516, False), (1024, 64, 1024, True)]),
    _case("relu_matmul", m=129, k=31, n=65, dtype="f32", call="device"),
    # ... of 16-bit operands that TMA cannot fetch
    _case("dot", m=65, k=77, n=131, dtype="bf16", transposed=False), _case("dot", m=200, k=45, n=99, dtype="f16", transposed=True),
    # tensor-core products: both tile heights, every width, K below and across a stage
    *(_case("dot", m=m, k=k, n=n, dtype=dt, transposed=t) for m, k, n, dt, t in
      [(33, 8, 8, "bf16", False), (129, 72, 136, "f16", True), (256, 64, 264, "bf16", True), (1000, 200, 2048, "bf16", False), (2304, 320, 4104, "bf16", True)]),
    # few rows: one and two row blocks, column blocks of every width, K of less than a group per warp
    *(_case("dot", m=m, k=k, n=n, dtype=dt, transposed=t) for m, k, n, dt, t in
      [(1, 8, 8, "bf16", False), (16, 40, 72, "f16", True), (17, 1032, 1000, "bf16", False), (32, 512, 4096, "bf16", True), (32, 2048, 2408, "f16", False)]),
    # ... by more columns than the lanes take in one round
    *(_case("dot", m=m, k=k, n=n, dtype=dt, transposed=t) for m, k, n, dt, t in
      [(1, 64, 4744, "bf16", False), (31, 72, 9480, "f16", True), (2, 4096, 9472, "bf16", False), (16, 4096, 9480, "bf16", True)]),
    # row pipelines and flat chains
    *(_case("norm_chain", rows=r, cols=n, dtype=dt) for r, n, dt in
      [(1, 128, "f32"), (149, 130, "bf16"), (64, 1023, "f16"), (300, 2048, "bf16"), (33, 4096, "f32")]),
    _case("int_chain", rows=1, cols=131), _case("int_chain", rows=601, cols=1025), _case("int_chain", rows=2048, cols=512),
    # store epilogues: GELU, its derivative, the update step, the loss sum
    _case("mlp", batch=72, d0=64, d1=136, d2=264, d3=72, dtype="bf16"), _case("mlp", batch=300, d0=64, d1=264, d2=520, d3=72, dtype="f16"), _case("mlp", batch=67, d0=33, d1=50, d2=21, d3=40, dtype="f32"),
    # attention between products; a decode step with its cache rows stored by the products
    _case("block", batch=3, seq=1100, heads=12, dtype="f16"), _case("block", batch=2, seq=65, heads=4, dtype="bf16"), _case("block", batch=1, seq=77, heads=4, dtype="f32"), _case("block", batch=1, seq=300, heads=2, dtype="f32"),
    # decode attention: fewer heads than lanes and more, whole stages of keys and one key past them, several heads per lane
    _case("decode", batch=1, cache=2047, heads=4, dtype="bf16"), _case("decode", batch=10, cache=600, heads=16, dtype="f16"), _case("decode", batch=32, cache=256, heads=5, dtype="bf16"),
    _case("decode", batch=1, cache=9000, heads=16, dtype="bf16"),
    _case("decode", batch=1, cache=64, heads=4, dtype="bf16"), _case("decode", batch=17, cache=301, heads=8, dtype="f16"), _case("decode", batch=3, cache=70, heads=4, dtype="f32"),
    _case("nbody", bodies=257, steps=2),
])
def test_planned_program(c):
    import perf.cases as cases
    state = cases.prepare(c, 5)
    args = [x.clone() for x in state["args"]]
    for _ in range(2):                            # the second run finds what the first one left behind
        outs = cases.run(state)
    torch.cuda.synchronize()
    assert state["lp"].Status()["code"] == 0 and state["lp"].stat("replanned") == 1
    tol = cases.tolerance(c)
    for got, want in zip(outs, _reference(c, args)):
        if tol == "exact":
            assert torch.equal(got, want)
            continue
        got, want = got.double(), want.double()
        assert torch.isfinite(got).all() and float((got - want).norm()) <= tol["rel"] * float(want.norm()) + 1e-30
        # ... and row by row, against the row and a typical one: a wrong row of many is lost in the whole
        if want.dim():
            rows, err = want.reshape(want.shape[0], -1).norm(dim=1), (got - want).reshape(want.shape[0], -1).norm(dim=1)
            assert bool((err <= 4 * tol["rel"] * (rows + rows.square().mean().sqrt())).all())


def _load(asm):
    import perf.cases as cases
    s = cases._runtime()
    return s, s["vm"].LoadedProgram.Load(s["rt"], s["vm"].VmProgram.Parse(asm.blob()))


def _execute(asm, args, runs=2):
    """The results of the program on these arguments (the last of `runs` runs: a later one finds what the first left behind)."""
    import perf.cases as cases
    s, lp = _load(asm)
    outs = [torch.empty(asm.dims[b], dtype=cases._TORCH[asm.bufs[b][1]], device="cuda") for b in asm.outputs]
    torch.cuda.synchronize()
    for _ in range(runs):
        lp.ExecuteDeviceAsync([a.data_ptr() for a in args], [o.data_ptr() for o in outs], s["stream"].cuda_stream)
    assert lp.Status()["code"] == 0
    return lp, outs


def _normal(shape, dtype, seed, scale=1.0, shift=0.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=gen, device="cuda") * scale + shift).to(dtype)


@pytest.mark.parametrize("rows, cols, dtype", [
    (4096, 1024, "f32"), (4096, 4096, "f32"), (150, 516, "f32"), (2000, 8192, "f32"), (700, 8196, "f32"), (4096, 4096, "bf16"), (700, 16384, "bf16")])
def test_residual_and_layer_norm(rows, cols, dtype):
    """Two staged operands per row: at the widths where the thread groups change, past the widest that is staged, and
    with enough rows on a lane that every buffer is used. Bound: a sum of squares is chains of at most 64 terms and a
    tree of 10, 74 x 2^-24 relative, half of that through the root, and the element's own few roundings (16-bit: half a
    step of 2^-8 per stored value, three of them, and the first changes what is normed)."""
    dt = getattr(torch, {"f32": "float32", "bf16": "bfloat16"}[dtype])
    x, y = _normal((rows, cols), dt, 1), _normal((rows, cols), dt, 2)
    g, b = _normal((cols,), dt, 3, 0.1, 1.0), _normal((cols,), dt, 4, 0.1)
    lp, (out,) = _execute(progs.residual_norm(rows, cols, dtype), [x, y, g, b])
    assert lp.stat("replanned") == 1
    s = (x + y).double()
    n = (s - s.mean(1, keepdim=True)) / torch.sqrt(s.var(1, unbiased=False, keepdim=True) + 1e-5)
    if dtype != "f32":
        n = n.to(dt).double()
    want = n * g.double() + b.double()
    tol = 4e-6 if dtype == "f32" else 2.0 ** -7
    assert bool(((out.double() - want).abs() <= tol * (1.0 + n.abs())).all())


@pytest.mark.parametrize("spec", [progs.REVERSED, progs.BLOCKED], ids=["reversed", "blocked"])
def test_product_through_an_operand_view(spec):
    """A view that is affine on neither side of a plain matrix; with a reversed axis the program keeps its own matmul."""
    M, K, N, dtype, dims, strides, off, elems = spec
    a, w = _normal((elems,), torch.float32, 1), _normal((K, N), torch.float32, 2)
    lp, (out,) = _execute(progs.viewed_product(*spec), [a, w])
    assert lp.stat("replanned") == (0 if min(strides) < 0 else 1)
    idx = sum(torch.arange(d).view([-1 if i == k else 1 for i in range(len(dims))]) * s for k, (d, s) in enumerate(zip(dims, strides))) + off
    ref = a.double()[idx.reshape(M, K).cuda()]
    # K products and sums of f32: K x 2^-24 of the sum of magnitudes
    assert bool(((out.double() - ref @ w.double()).abs() <= K * 2.0 ** -24 * (ref.abs() @ w.double().abs())).all())


@pytest.mark.parametrize("what", ["product", "residual", "gelu", "both"])
@pytest.mark.parametrize("mnk", [(300, 264, 64), (16, 72, 64), (40, 33, 45)], ids=["gemm", "skinny", "sgemm"])
def test_product_converted_after_a_16_bit_value(what, mnk):
    """What the program holds in bf16 has bf16's values after the convert to f32. Small integers: products and sums are exact in
    f32, so the roundings to bf16 are all there is and the bits are known (but for GELU, whose result has to be a bf16 number)."""
    M, N, K = mnk
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, w, x = (torch.randint(-8, 9, s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((M, K), (K, N), (M, N)))
    lp, (out,) = _execute(progs.widened_product(M, K, N, "bf16", what), [a, w, x])
    assert lp.stat("replanned") == 1
    y = (a.double() @ w.double()).to(torch.bfloat16)
    assert float(y.abs().max()) > 256                  # beyond 8 bits: it had to be rounded
    if what in ("residual", "both"):
        y = (x.double() + y.double()).to(torch.bfloat16)
    assert torch.equal(out, out.to(torch.bfloat16).float())
    if what in ("gelu", "both"):
        want = _gelu(y.double())
        assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())      # half a step of bf16, and gelu_tanh's own error
    else:
        assert torch.equal(out, y.float())


@pytest.mark.parametrize("what", ["product", "residual", "gelu", "kept", "grad", "step", "loss", "times", "wide", "both"])
@pytest.mark.parametrize("M, K, N, dtype, transposed", [
    (33, 64, 8, "bf16", False), (128, 72, 104, "f16", False), (129, 200, 264, "bf16", False), (300, 1096, 520, "f16", True), (200, 64, 99, "bf16", True),
    (2100, 136, 1032, "bf16", False), (9600, 64, 4104, "f16", False)])
def test_store_epilogues_at_the_edges_of_tiles(what, M, K, N, dtype, transposed):
    """One and two halves of 128 rows, column chunks that end inside a tile, rows that are no whole 16-byte words (the general
    form), rings of 3 to 8 stages that wrap. Small integers: products and sums are exact in f32, so the roundings to the 16-bit type
    are all there is and the bits are known (but for GELU: a step of the type, and gelu_tanh's own error; its derivative alike, of which
    the product takes a multiple; and the sum of squares, added in f32 by chains of at most 64 terms, 256 chunks and a tree)."""
    dt = {"bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, w, x = (torch.randint(-3, 4, s, generator=gen, device="cuda").to(dt) for s in ((M, K), (N, K) if transposed else (K, N), (M, N)))
    lp, outs = _execute(progs.product_then(M, K, N, dtype, what, transposed), [a, w, x.float() if what == "wide" else x])
    assert lp.stat("tensor_core_matmuls") == 1
    y = (a.double() @ (w.T if transposed else w).double()).float()
    if what == "step":
        assert torch.equal(outs[0], (x.float() - y * torch.tensor(1e-3, device="cuda")).to(dt))
    y = y.to(dt)
    if what in ("times", "wide"):
        assert torch.equal(outs[0], y * x if what == "times" else y.float() + x.float())
    if what == "loss":
        d = y.float() - x.float()
        total, scaled = outs
        assert torch.equal(scaled, (d * torch.tensor(2.0 / (M * N), device="cuda")).to(dt))
        want = float((d.double() ** 2).sum())
        assert abs(float(total) - want) <= 384 * 2.0 ** -24 * want
    if what == "grad":
        z = x.double().requires_grad_()
        slope, = torch.autograd.grad(_gelu(z).sum(), z)
        want = y.double() * slope
        assert bool(((outs[0].double() - want).abs() <= (2.0 ** -8 if dtype == "bf16" else 2.0 ** -11) * want.abs() + 2e-6 * y.double().abs()).all())
    if what in ("product", "kept", "both"):
        assert torch.equal(outs[0], y)
    if what in ("residual", "both"):
        assert torch.equal(outs[-1], (x.float() + y.float()).to(dt))
    if what in ("gelu", "kept"):
        want = _gelu(y.double())
        assert bool(((outs[-1].double() - want).abs() <= (2.0 ** -8 if dtype == "bf16" else 2.0 ** -11) * want.abs() + 1e-6).all())


@pytest.mark.parametrize("bodies", [258, 400])
def test_bodies_whose_squared_distance_overflows(bodies):
    """Two clusters 1e20 apart: between them the squared distance is infinite in f32 and the weight 0, as pow(inf, -1.5) is;
    inside each the accelerations are those of the cluster alone."""
    import perf.cases as cases
    c = {"kind": "nbody", "bodies": bodies, "steps": 1}
    gen = torch.Generator(device="cuda").manual_seed(2)
    pos = torch.rand((bodies, 3), generator=gen, device="cuda") * 2 - 1
    vel, mass = torch.zeros((bodies, 3), device="cuda"), torch.rand(bodies, generator=gen, device="cuda") + 0.5
    half = bodies // 2
    pos[half:, 0] = 1e20                               # (their own x distances are 0: 1e20 swallows the rest)
    lp, (p1, v1) = _execute(cases._BUILD["nbody"](c), [pos, vel, mass])
    assert lp.stat("pairs") == 4
    for s in (slice(0, half), slice(half, bodies)):
        near = pos[s].clone()
        if s.start:
            near[:, 0] = 0.0
        want = _reference(c, [near, vel[s], mass[s]])
        got = p1[s].clone()
        if s.start:
            got[:, 0] -= 1e20
        for g, w in ((got, want[0]), (v1[s], want[1])):
            assert torch.isfinite(g).all() and float((g.double() - w).norm()) <= 1e-5 * float(w.norm())
    # a NaN is no infinite distance: it reaches everyone
    pos[3, 1] = float("nan")
    _, (p1, v1) = _execute(cases._BUILD["nbody"](c), [pos, vel, mass])
    assert bool(torch.isnan(v1[:half]).any(1).all())


@pytest.mark.parametrize("n, steps, after", [(64, (0.5, 0.25), 0), (301, (0.5, 0.25, 0.125), 0), (1000, (0.0, 0.5, 0.25), 20), (257, (0.5, 0.0), 24)])
def test_independent_evaluations(n, steps, after):
    """Evaluations that share phases, and positions made in another one's tail. f32 from the same positions: a difference, a few
    products and the root per pair (2^-20), sums of n terms as chains of at most n / 32 and a tree."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    x, v = (torch.rand((n, 3), generator=gen, device="cuda") * 2 - 1 for _ in range(2))
    mass = torch.rand(n, generator=gen, device="cuda") + 0.5
    lp, outs = _execute(progs.evaluations(n, steps, after), [x, v, mass])
    at, acc = [v * s + x for s in steps], outs[:len(steps)]
    if after:
        moved, last = outs[-2:]
        assert torch.equal(moved, (acc[0] + x) * (-1.0) ** (after - 1))
        at, acc = at + [moved], acc + [last]
    assert lp.stat("replanned") == 1 and lp.stat("pairs") == len(at) == len(acc)
    for out, p in zip(acc, at):
        p = p.double()
        d = p[None] - p[:, None]
        f = d * ((d * d).sum(2) + 1e-4).pow(-1.5).mul(mass.double()[None])[..., None]
        assert bool(((out.double() - f.sum(1)).abs() <= (n / 32 + 64) * 2.0 ** -24 * f.abs().sum(1)).all())


@pytest.mark.parametrize("H, T, C, hd", [(40, 64, 64, 64), (12, 129, 129, 64), (41, 33, 100, 64), (20, 70, 131, 40), (22, 64, 67, 128), (6, 300, 301, 200), (3, 33, 70, 64)])
def test_masked_values_do_not_reach_the_rows_that_mask_them(H, T, C, hd):
    """Causal attention on the CUDA cores: a NaN, or an infinity, in the V row of key c shows in the query rows that see c and
    in no other, wherever c lies in its chunk of 64. f32 in another order than torch's: C x 2^-24, and the exponentials."""
    q, q0, k, v = (_normal(s, torch.float32, i) for i, s in enumerate(((H, T, hd), (H, T, hd), (H, hd, C), (H, C, hd))))
    seen = torch.arange(C, device="cuda")[None, :] <= torch.arange(T, device="cuda")[:, None] + C - T
    s = ((q + q0).double() @ k.double() / hd ** 0.5).masked_fill(~seen, float("-inf"))
    want = torch.softmax(s, -1) @ v.double()
    for c in sorted({C - T, C - T + 1, C - T + 2, C - 1, C - 2, min(C - 1, 63), min(C - 1, 64)}):
        bad = v.clone()
        bad[:, c] = float("nan")
        bad[0, c] = float("inf")
        lp, (out,) = _execute(progs.attention_of_sums(H, T, C, hd, "f32", True), [q, q0, k, bad])
        assert lp.stat("replanned") == 1
        clean = ~seen[:, c]
        assert bool((~torch.isfinite(out[:, ~clean])).all())
        assert bool(((out[:, clean].double() - want[:, clean]).abs() <= 1e-5 * (1.0 + want[:, clean].abs())).all())


@pytest.mark.parametrize("mkn", [((64, 8192, 64), (1024, 512, 1024)), ((100, 512, 256), (400, 128, 100)), ((64, 64, 640), (400, 1024, 512), (256, 2048, 640)),
                                 ((2000, 64, 2000), (1500, 100, 3000))], ids=str)
def test_products_side_by_side(mkn):
    """f32: K products and sums, K x 2^-24 of the sum of magnitudes."""
    args = [_normal(s, torch.float32, i) for M, K, N in mkn for i, s in enumerate(((M, K), (K, N)))]
    lp, outs = _execute(progs.products("f32", *mkn), args)
    assert lp.stat("replanned") == 1 and lp.stat("planned_phases") == 1
    for out, a, w in zip(outs, args[::2], args[1::2]):
        a, w = a.double(), w.double()
        assert bool(((out.double() - a @ w).abs() <= a.shape[1] * 2.0 ** -24 * (a.abs() @ w.abs())).all())


def _attention(q, k, v, causal):
    """Attention in float64, sum p |v|, and which keys a row sees."""
    T, C = q.shape[1], v.shape[1]
    seen = torch.arange(C, device="cuda")[None, :] <= torch.arange(T, device="cuda")[:, None] + (C - T if causal else C)
    p = torch.softmax((q.double() @ k.double() / q.shape[2] ** 0.5).masked_fill(~seen, float("-inf")), -1)
    return p @ v.double(), p @ v.double().abs(), seen


# What the roundings allow: P and the result to half a step each, 2^-8 of a bf16 value and 2^-11 of an f16 one; a score's f32 sum of 64
# products (4 x: the tensor cores' own order and truncation); f16: the denormal steps of P, whose largest value in a row is at least 1.
def _attention_bound(q, k, v, mag):
    score = 64 * 2.0 ** -22 * float((q.double().abs() @ k.double().abs()).max()) / 8
    return ((2.0 ** -7 if q.dtype == torch.bfloat16 else 2.0 ** -10) + 2 * score) * mag + v.shape[1] * 2.0 ** -25 * float(v.abs().max()) + 1e-6


@pytest.mark.parametrize("trips", [0, 2], ids=["drawn", "split"])
@pytest.mark.parametrize("H, T, C, dtype, causal", [
    (4, 320, 320, "bf16", True), (5, 130, 1104, "f16", False), (3, 300, 1111, "bf16", True), (230, 129, 300, "bf16", True), (75, 129, 129, "f16", True), (1, 16, 64, "bf16", False)])
def test_attention_whose_row_maxima_grow(H, T, C, dtype, causal, trips, monkeypatch):
    """Scores that grow by up to 2^12 from one block of 64 keys to the next (rows by turns: none, 2^6, 2^12, and shrinking), so that
    the accumulators are rescaled at every block of some rows, at every other of others, in no row of a warp or in some. Tiles
    drawn from a counter (an attention that runs once) and split by rows (the body of a loop); re-planned and as scheduled."""
    dt = {"bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    u = torch.full((64,), 0.125, device="cuda")
    row, key = torch.arange(T, device="cuda"), torch.arange(C, device="cuda")
    lean = torch.tensor([0.0, 2.0, 4.0, -4.0], device="cuda")[torch.where(row % 96 < 32, row % 4, row // 32 % 4)]
    q = (_normal((H, T, 64), torch.float32, 1) + lean[None, :, None] * u).to(dt)
    k = (_normal((H, 64, C), torch.float32, 2, 0.5) + 16.6 * (key // 64)[None, None, :] * u[:, None]).to(dt)
    v, zero = _normal((H, C, 64), dt, 3), torch.zeros_like(q)
    want, mag, _ = _attention(q, k, v, causal)
    bound = _attention_bound(q, k, v, mag)
    for replanned in (1, 0):
        if not replanned:
            monkeypatch.setenv("B2VM_NO_REPLAN", "1")
        by_key = C % 8 != 0                # (rows of [64, C] start on 16-byte boundaries, or the tensor cores are not used)
        lp, (out,) = _execute(progs.attention_of_sums(H, T, C, 64, dtype, causal, trips, by_key), [q, zero, k.mT.contiguous() if by_key else k, v])
        assert lp.stat("replanned") == replanned and lp.stat("tensor_core_flash") == 1
        assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("C, causal", [(333, True), (336, False), (200, True)])
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
def test_attention_with_nan_and_infinite_scores(dtype, C, causal):
    """A NaN in a query row shows in that row alone; a NaN or an infinite score of a key in the rows that see the key and no other;
    a score of minus infinity takes the key out."""
    H, T = 3, 200
    dt = {"bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    q, k, v = _normal((H, T, 64), dt, 1), _normal((H, 64, C), dt, 2), _normal((H, C, 64), dt, 3)
    q[:, :, 7] = q[:, :, 7].abs() + 0.5
    zero = torch.zeros_like(q)
    want, mag, seen = _attention(q, k, v, causal)
    bound = _attention_bound(q, k, v, mag)

    def run(q, k):
        by_key = C % 8 != 0
        lp, (out,) = _execute(progs.attention_of_sums(H, T, C, 64, dtype, causal, 0, by_key), [q, zero, k.mT.contiguous() if by_key else k, v])
        assert lp.stat("tensor_core_flash") == 1
        return out
    bad = q.clone()
    bad[1, 131, 9] = float("nan")
    out, hit = run(bad, k), torch.zeros((H, T), dtype=torch.bool, device="cuda")
    hit[1, 131] = True
    assert bool(torch.isnan(out[hit]).all()) and bool(((out.double() - want).abs() <= bound)[~hit].all())
    for c in (0, 63, 64, 150, C - 1):
        for x in (float("nan"), float("inf")):
            bad = k.clone()
            bad[2, 7, c] = x
            out, hit = run(q, bad), torch.zeros((H, T), dtype=torch.bool, device="cuda")
            hit[2] = seen[:, c]
            assert bool(torch.isnan(out[hit]).all()) and bool(((out.double() - want).abs() <= bound)[~hit].all())
        if c:                      # (every row sees key 0 at least)
            bad = k.clone()
            bad[:, 7, c] = float("-inf")
            want_c, mag_c, _ = _attention(q, bad, v, causal)
            assert bool(((run(q, bad).double() - want_c).abs() <= _attention_bound(q, k, v, mag_c)).all())


@pytest.mark.parametrize("what, total", [
    (("mul", "add", "gelu"), False), (("mul", "add", "gelu"), True), (("add",), False), (("mul",), True), (("gelu",), False), (("mul", "gelu"), False), (("res", "gelu"), True),
    (("res", "mul", "add"), False), (("res",), True), ((), True)], ids=lambda v: "-".join(v) if isinstance(v, tuple) else "sum" if v else "")
@pytest.mark.parametrize("rows, cols, dtype", [(1, 640, "f32"), (1, 256, "f32"), (1, 256, "bf16"), (700, 1024, "f32"), (333, 130, "f32"), (150, 4096, "bf16"), (64, 1023, "f16"), (2048, 512, "bf16"), (77, 8192, "f32")])
def test_pipelines_without_a_norm(what, total, rows, cols, dtype):
    """Every stage on its own and together, in rows and in pieces of a flat list: a value differs from the same stages rounded one
    by one in float64 by a step of its type at most (GELU's approximation may turn a rounding), f32 by a few 2^-23; the sum
    by the f32 additions of a lane's chain and the tree over them."""
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    x = _normal((rows, cols), dt, 1)
    args, cur = [x], x.double()
    for i, w in enumerate(what):
        if w == "gelu":
            cur = _gelu(cur)
        else:
            args.append(_normal((rows, cols) if w == "res" else (cols,), dt, 2 + i, *((0.1, 1.0) if w == "mul" else (1.0,))))
            cur = cur * args[-1].double() if w == "mul" else cur + args[-1].double()
        cur = cur.to(dt).double()
    lp, outs = _execute(progs.stages(rows, cols, dtype, what, total), args)
    step = {"f32": 2.0 ** -21, "bf16": 2.0 ** -7, "f16": 2.0 ** -10}[dtype]
    if what:
        got = outs[0].double()
        assert bool(((got - cur).abs() <= step * cur.abs() + (2e-6 if "gelu" in what else 2.0 ** -24)).all())
    if total:
        # of what was stored (bit for bit), in f32: chains of at most rows x cols / (148 x 512) + 8, then trees of 9 and 8
        kept = (outs[0] if what else x).double()
        bound = (rows * cols / (148 * 512) + 64) * 2.0 ** -24 * float(kept.abs().sum())
        assert abs(float(outs[-1]) - float(kept.sum())) <= bound


@pytest.mark.parametrize("cols, dtype", [(64, "f32"), (100, "f32"), (640, "bf16")])
def test_reciprocal_roots_and_reciprocals_against_the_exact_ones(cols, dtype):
    """Rows v, 0, 0, ... normed without an epsilon come out as sqrt(cols), rows of equal elements through a softmax as 1 / cols,
    whatever v's magnitude: 1 / sqrt(x) and 1 / x by one Newton step on the approximations. Bound for f32: 2 units for the step
    (CUDA documents 2 ulp and 1 ulp for the approximations alone), and the products' own."""
    import perf.cases as cases
    dt = {"f32": torch.float32, "bf16": torch.bfloat16}[dtype]
    rows = 4096
    lo, hi = (-17.0, 17.0) if dtype == "f32" else (-15.0, 15.0)
    v = (10.0 ** torch.linspace(lo, hi, rows, device="cuda", dtype=torch.float64)).to(dt)
    x = torch.zeros((rows, cols), dtype=dt, device="cuda")
    x[:, 3] = v
    ones = torch.ones(cols, dtype=dt, device="cuda")
    p = cases._Assembler(148)
    xi, g = p.input((rows, cols), dtype), p.input((cols,), dtype)
    p.output(progs.rms_norm(p, xi, g, rows, cols, dtype, eps=0.0), (rows, cols))
    lp, (out,) = _execute(p, [x, ones])
    assert lp.stat("replanned") == 1
    want = cols ** 0.5
    step = 6 * 2.0 ** -24 if dtype == "f32" else 2.0 ** -8
    assert bool(((out[:, 3].double() - want).abs() <= step * want).all()) and int((out != 0).sum()) == rows
    if dtype == "f32":
        x = (v / v.max() * 80.0)[:, None].expand(rows, cols).contiguous()
        p = cases._Assembler(148)
        p.output(p.rows(cases._SOFTMAX, p.input((rows, cols), dtype), rows, cols), (rows, cols))
        lp, (out,) = _execute(p, [x])
        assert lp.stat("replanned") == 1 and bool(((out.double() * cols - 1).abs() <= 4 * 2.0 ** -24).all())


def test_norm_of_rows_whose_mean_square_is_denormal():
    """Powers of two down to 2^-70, no epsilon: the mean square is exact down to 2^-146 and its root finite."""
    import perf.cases as cases
    rows, cols = 148 * 4, 64
    x = torch.zeros((rows, cols), device="cuda")
    x[:, 5] = 2.0 ** -(60 + torch.arange(rows, device="cuda") % 11)
    p = cases._Assembler(148)
    xi, g = p.input((rows, cols), "f32"), p.input((cols,), "f32")
    p.output(progs.rms_norm(p, xi, g, rows, cols, "f32", eps=0.0), (rows, cols))
    lp, (out,) = _execute(p, [x, torch.ones(cols, device="cuda")])
    assert lp.stat("replanned") == 1
    assert bool(((out[:, 5].double() - 8).abs() <= 8 * 4 * 2.0 ** -23).all())      # 2 ulp of the approximation, and the product


@pytest.mark.parametrize("m, k, n, transposed", [(33, 4096, 16000, True), (33, 512, 11008, True), (100, 1024, 16000, False), (33, 64, 8192, True)])
def test_products_of_one_tile_per_lane_with_cold_caches(m, k, n, transposed):
    """A lane's last product ends the launch, and nothing of it may still be under way: many launches, code and operands out of L2."""
    import perf.cases as cases
    st = cases.prepare(dict(kind="dot", m=m, k=k, n=n, dtype="bf16", transposed=transposed), 3)
    assert st["lp"].stat("replanned") == 1 and st["lp"].stat("tensor_core_matmuls") == 1
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    a, w = (x.double() for x in st["args"])
    want = a @ (w.T if transposed else w)
    for i in range(40):
        flush.fill_(i)
        torch.cuda.synchronize()
        (out,) = cases.run(st)
        assert st["lp"].Status()["code"] == 0
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + k * 2.0 ** -24 * (a.abs() @ (w.T if transposed else w).abs())).all())


@pytest.mark.parametrize("m, heads", [(300, 0), (0, 4)])
def test_arguments_and_results_at_other_addresses_every_call(m, heads):
    """Operands that are arguments are fetched through tensor maps made anew when an address changes: calls that alternate between
    two sets of buffers, with nothing in between, each see their own."""
    import perf.cases as cases
    c = dict(kind="dot", m=m, k=264, n=520, dtype="bf16", transposed=False) if m else dict(kind="block", batch=1, seq=130, heads=heads, dtype="bf16")
    a, b = cases.prepare(c, 1), cases.prepare(c, 2)
    want = []
    for st in (a, b):
        cases.run(st)
        assert st["lp"].Status()["code"] == 0
        want.append([o.clone() for o in st["outs"]])
    lp, stream = a["lp"], a["stream"]
    for _ in range(20):
        for st in (a, b):
            for o in st["outs"]:
                o.zero_()
        torch.cuda.synchronize()
        for st in (a, b, a, b):
            lp.ExecuteDeviceAsync(st["in_ptr"], st["out_ptr"], stream)
        assert lp.Status()["code"] == 0
        for st, w in zip((a, b), want):
            assert all(torch.equal(o, x) for o, x in zip(st["outs"], w))
