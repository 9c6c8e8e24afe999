"""What the re-planner makes of a program, on the host: the planner and the table builder alone, without a device."""
from __future__ import annotations

import glob
import gzip
import importlib
import itertools
import json
import math
import os
import re
import subprocess

import pytest

from conftest import ROOT
import perf.cases as cases
import plan_programs as progs

CSRC = os.path.join(ROOT, "pjrt-ocl_b200", "csrc")
FUSE_ROWS, PAIRS, GEMM, SGEMM, SKINNY, MMA = 33, 34, 35, 37, 38, 1
ON, RES, LN, MUL, ADD, GELU, CARRY = 1, 2, 4, 16, 32, 64, 256           # row pipeline stages (plan_format.h)
F32, BF16, QUANT0, EPI_GELU, EPI_RES = 0, 7, 1, 2, 16


@pytest.fixture(scope="session")
def plan(tmp_path_factory):
    """blob -> the plan's facts."""
    d = tmp_path_factory.mktemp("plan")
    exe = str(d / "plan_probe")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, os.path.join(ROOT, "tests", "adapter", "plan_probe.cc"),
                    *(os.path.join(CSRC, f) for f in ("vmprog.cc", "loader.cc", "replan.cc")), "-o", exe], check=True)

    def run(blob, lanes=148):
        (d / "blob").write_bytes(blob)
        r = subprocess.run([exe, str(d / "blob"), str(lanes)], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return json.loads(r.stdout)
    return run


@pytest.mark.parametrize("rows, cols", [(149, 516), (8192, 1024), (4096, 4096), (16384, 768), (2000, 8192), (700, 8196), (300, 16384), (40, 16384)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_staged_rows_of_a_pipeline_fit_the_shared_memory(plan, rows, cols, dtype):
    (t,) = [t for t in plan(progs.residual_norm(rows, cols, dtype).blob())["tasks"] if t["op"] == FUSE_ROWS]
    assert t["stage"] <= t["room"]
    # f32 rows past 512 threads x 16 elements leave the row pipelines; the others are still on them
    assert (t["pipe"] & (RES | LN | MUL | ADD)) == (0 if dtype == "f32" and cols > 8192 else RES | LN | MUL | ADD)


def test_reversed_operand_views_stay_off_the_cuda_core_product(plan):
    """Its offsets are unsigned: a part of a place that is negative would be read 2^32 elements too far."""
    ok = plan(progs.viewed_product(*progs.BLOCKED).blob())
    assert [t["viewed"] for t in ok["tasks"] if t["op"] == SGEMM] == [[1, 0]]
    assert not [t for t in plan(progs.viewed_product(*progs.REVERSED).blob())["tasks"] if t["op"] in (SGEMM, SKINNY)]
    # reversed along k, beside a plain second axis; and a plain reversed k
    for dims, strides, off in (((2, 8, 64), (512, 64, -1), 63), ((2, 8, 2, 32), (512, 64, -32, 1), 32), ((16, 64), (64, -1), 63)):
        assert not [t for t in plan(progs.viewed_product(16, 64, 24, "f32", dims, strides, off, 1024).blob())["tasks"] if t["op"] in (SGEMM, SKINNY)]


@pytest.mark.parametrize("what, flags, dt1", [("product", QUANT0, F32), ("residual", QUANT0 | EPI_RES, BF16), ("gelu", QUANT0 | EPI_GELU, BF16),
                                              ("both", QUANT0 | EPI_RES, BF16)])
@pytest.mark.parametrize("mnk", [(256, 256, 64), (16, 64, 64), (40, 33, 45)])
def test_products_keep_the_roundings_of_what_they_hand_on(plan, what, flags, dt1, mnk):
    """A value that the program holds in 16 bits leaves a store epilogue in 16 bits, or rounded."""
    M, N, K = mnk
    tasks = plan(progs.widened_product(M, K, N, "bf16", what).blob())["tasks"]
    got = [(q["epi"], q["dt1"]) for t in tasks for q in t.get("prob", [t]) if "epi" in q]
    assert got == [(flags, dt1)]


@pytest.mark.parametrize("lanes, device, planned", [(74, 148, False), (75, 148, True), (66, 132, False), (66, 131, True), (148, 148, True)])
def test_schedules_for_half_the_device_stay_side_by_side(plan, lanes, device, planned):
    assert plan(progs.residual_norm(600, 256, "f32", lanes).blob(), device)["planned"] == planned


def test_asynchronous_copies_follow_a_fence_over_the_workspace():
    """Every function that sets up barriers for copies into shared memory first fences the asynchronous proxy against what the
    lane's entry before wrote there by ordinary stores (no run shows a missing fence for certain: the source does)."""
    n = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "ops_*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"fence_mbar_init\(\)", text):
            n += 1
            # a fence by all threads, then the barrier that the thread which issues the copies passes
            before, after = text[:m.start()], text[m.start():]
            fenced = before.rfind("fence_proxy_async_smem()")
            first = after.index("__syncthreads()")
            near = fenced >= 0 and "__global__" not in before[fenced:] and "static __device__" not in before[fenced:] and "__syncthreads()" in before[fenced:]
            assert near or "fence_proxy_async_smem()" in after[:first], (os.path.basename(path), before.count("\n"))
    assert n >= 6


def committed(name):
    return gzip.open(os.path.join(ROOT, "pjrt-ocl_b200", "programs", name + ".vmprog.gz")).read()


def test_chains_without_a_norm_are_row_pipelines(plan):
    (t,) = plan(committed("c2_stage_affine_gelu_f32"))["tasks"]
    assert t["pipe"] == ON | MUL | ADD | GELU
    (t,) = plan(committed("c2_stage_sum_f32"))["tasks"]
    assert t["pipe"] == ON | CARRY


@pytest.mark.parametrize("n, dtype, ops, kept", [
    (131, "i32", (cases._ADD, cases._XOR, cases._MAX), True), (33550001, "i32", (cases._ADD, cases._XOR, cases._MAX), False),
    (33550000, "i32", (cases._ADD, cases._XOR, cases._MAX), True), (400001, "bf16", (cases._ADD,), True), (4000001, "bf16", (cases._ADD,), False),
    (33550000, "bf16", (cases._ADD, cases._MUL), False), (8192 * 4096, "bf16", (cases._GELU,), True), (33550001, "f32", (cases._TANH, cases._MUL), False)])
def test_long_chains_that_only_the_step_interpreter_runs_keep_their_schedule(plan, n, dtype, ops, kept):
    p = plan(progs.flat(n, dtype, ops).blob())
    assert p["planned"] and p["gains"] == kept


def test_norm_chains_and_products_keep_their_plans(plan):
    for c in cases.listed():
        if c["kind"] != "nbody":
            assert plan(cases._BUILD[c["kind"]](c).blob())["gains"], c["name"]
    # an odd width: the interpreter, but instead of four passes
    assert plan(cases._BUILD["norm_chain"]({"rows": 8192, "cols": 4095, "dtype": "f32"}).blob())["gains"]
    # a lone sum of a length that no piece divides: the tile op streams it faster
    assert not plan(progs.stages(8191, 4095, "f32", (), True).blob())["gains"]


def test_products_beside_large_moves_get_their_lanes(plan):
    """The decode step that copies its caches: three products share a phase with the copies. They share the lanes among
    themselves as they would alone, and the copies are cut evenly over all."""
    tasks = plan(committed("c5_decode_bf16"))["tasks"]
    qkv = [t for t in tasks if t["op"] == SKINNY and t["mnk"] == [32, 1024, 1024]][:3]
    for t in qkv:
        assert len({lane for lane, _, _ in t["cut"]}) >= 32                 # 32 tiles of 32 columns each
    lanes = [lane for t in qkv for lane, _, _ in t["cut"]]
    assert len(lanes) == len(set(lanes))
    moves = [t for t in tasks if t["op"] in (2, 6) and max(hi for _, _, hi in t["cut"]) >= 2 * 148]
    assert len(moves) == 3
    for t in moves:
        per = [hi - lo for _, lo, hi in t["cut"]]
        assert len(per) == 148 and max(per) - min(per) <= 1


def test_tensor_core_ops_end_with_no_commit_under_way():
    """Every op whose products free its stages by a commit waits for the last of them before its barriers go: an arrival on an
    invalidated barrier, or in a CTA that has left, is a fault that a run shows once in many."""
    n = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "ops_*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        if "tc_commit(" not in text:
            continue
        n += 1
        assert text.rindex("tc_drain(") < text.rindex("mbar_inval("), os.path.basename(path)
    assert n == 3


@pytest.mark.parametrize("rows, cols, dtype, kept", [
    (8192, 2048, "f32", True), (8192, 2052, "f32", False), (8192, 4096, "bf16", False), (8192, 4094, "f32", True), (4096, 6912, "f32", False),
    (4096, 8192, "f32", True), (4096, 8192, "bf16", False), (2048, 13824, "bf16", False), (2048, 16384, "bf16", True), (64, 4096, "f32", True)])
def test_lone_norms_and_sums_stay_where_the_tile_op_is_faster(plan, rows, cols, dtype, kept):
    for softmax in (False, True):
        assert plan(progs.lone_norm(rows, cols, dtype, softmax).blob())["gains"] == kept
    assert plan(progs.stages(rows, cols, dtype, (), True).blob())["gains"] is False
    assert plan(progs.stages(rows, cols, dtype, ("gelu",), True).blob())["gains"]


def test_short_lone_sums_keep_their_plan(plan):
    assert plan(progs.stages(64, 128, "f32", (), True).blob())["gains"]


@pytest.mark.parametrize("m, k, n, transposed, op", [
    (32, 1024, 4736, False, SKINNY), (32, 1024, 4744, False, GEMM), (32, 1024, 4744, True, GEMM), (1, 4096, 9472, False, SKINNY), (5, 4096, 9472, False, GEMM),
    (1, 4096, 9480, False, GEMM), (16, 4096, 18944, True, SKINNY), (17, 4096, 9472, True, GEMM), (16, 4096, 18952, True, GEMM), (1, 2048, 9472, True, GEMM), (1, 2048, 9472, False, SKINNY), (1, 2040, 9472, False, GEMM)])
def test_few_rows_by_many_columns(plan, m, k, n, transposed, op):
    (t,) = plan(cases._BUILD["dot"](dict(m=m, k=k, n=n, dtype="bf16", transposed=transposed)).blob())["tasks"]
    assert t["op"] == op


@pytest.mark.parametrize("n", [64, 4096])
@pytest.mark.parametrize("steps, phases, others", [
    ((0.5, 0.25), 2, 2), ((0.5, 0.25, 0.125), 2, 3),                 # all positions side by side, then all evaluations
    ((0.0, 0.5), 2, 0), ((0.5, 0.0), 2, 0), ((0.0, 0.5, 0.25), 2, 0)])       # positions in the tail of the one that waits for none
def test_independent_evaluations_are_all_fused(plan, n, steps, phases, others):
    p = plan(progs.evaluations(n, steps).blob())
    run = [t["op"] for t in p["tasks"] if t["cut"]]
    assert p["gains"] and p["phases"] == phases and run.count(PAIRS) == len(steps) and run.count(FUSE_ROWS) == len(run) - len(steps) == others


@pytest.mark.parametrize("after, others", [(22, 0), (23, 1), (24, 1)])
def test_an_evaluations_own_tail_comes_before_other_evaluations_positions(plan, after, others):
    """A tail holds 24 ops: its own, and if they fit the two that make the other evaluation's positions. One of its own left out
    would be a phase of its own, for the evaluation that waits for it."""
    p = plan(progs.evaluations(64, (0.0, 0.5), after).blob())
    run = [t["op"] for t in p["tasks"] if t["cut"]]
    assert run.count(PAIRS) == 3 and len(run) == 3 + others and p["phases"] == 2


def test_an_rk4_step_is_four_evaluations(plan):
    p = plan(cases._BUILD["nbody"]({"bodies": 4096, "steps": 10}).blob())
    run = [t["op"] for t in p["tasks"] if t["cut"]]
    assert p["phases"] == 5 and run == [FUSE_ROWS, FUSE_ROWS] + [PAIRS] * 4


# a tile's rows and columns, slices of K and share of the issue rate, by shape, and its time, as Planner::SgShape has them
SGEMM_SHAPES = [(128, 64, 4, 0.75), (64, 64, 8, 0.75), (64, 32, 8, 0.6), (32, 32, 8, 0.45), (16, 16, 8, 0.2)]


def _sgemm_tiles(t):
    (m, n, k), (tm, tn, slices, rate) = t["mnk"], SGEMM_SHAPES[t["shape"]]
    return -(-m // tm) * -(-n // tn), max(k * tm * tn / (128 * rate), math.ceil(-(-k // 16) / slices) * 700.0) + 1500.0 + tm * tn * 0.15


@pytest.mark.parametrize("mkn", [
    ((512, 512, 512),) * 3, ((64, 8192, 64), (1024, 512, 1024)), ((777, 512, 100), (1024, 64, 256)), ((100, 512, 256), (400, 128, 100)),
    ((777, 2048, 100), (100, 256, 1024), (400, 64, 64)), ((400, 256, 1024), (777, 512, 1024), (512, 128, 256))], ids=str)
def test_products_side_by_side_share_the_lanes_by_whole_tiles(plan, mkn):
    """Lanes of their own, none without a tile, and no split of the lanes whose busiest one is done sooner."""
    tasks = [t for t in plan(progs.products("f32", *mkn).blob())["tasks"] if t["op"] == SGEMM]
    lanes = [lane for t in tasks for lane, _, _ in t["cut"]]
    tiles, cost = zip(*map(_sgemm_tiles, tasks))
    own = [len(t["cut"]) for t in tasks]
    assert len(tasks) == len(mkn) and len(lanes) == len(set(lanes)) and len(lanes) == min(148, sum(tiles))
    assert all(sorted(c[1:] for c in t["cut"]) == [[i, n] for i in range(n)] and n <= k for t, n, k in zip(tasks, own, tiles))

    def last(split):
        return max(c * -(-k // n) for c, k, n in zip(cost, tiles, split))
    splits = ((*s, 148 - sum(s)) for s in itertools.product(range(1, 148), repeat=len(mkn) - 1) if sum(s) < 148)
    assert last(own) <= min(map(last, splits)) * (1 + 1e-12)


def test_products_with_tiles_for_everybody_are_spread_over_all_lanes(plan):
    """Whatever the cost model makes of them."""
    for t in plan(progs.products("f32", (4096, 256, 4096), (2048, 1024, 2048)).blob())["tasks"]:
        assert sorted(lane for lane, _, _ in t["cut"]) == list(range(148))


# ops_gemm.cuh: an epilogue that is compiled for its steps (+ 16: of f16), 0 the general one
FORMS = {"product": 1, "gelu": 2, "kept": 2, "residual": 3, "grad": 4, "step": 5, "loss": 6, "times": 0, "wide": 0, "both": 0}


@pytest.mark.parametrize("what", FORMS)
@pytest.mark.parametrize("M, K, N, dtype, transposed, general", [
    (33, 64, 8, "bf16", False, False), (129, 200, 264, "f16", False, False), (200, 64, 99, "bf16", True, True), (9600, 64, 4104, "bf16", False, False)])
def test_epilogues_run_in_the_form_for_their_steps(plan, what, M, K, N, dtype, transposed, general):
    p = plan(progs.product_then(M, K, N, dtype, what, transposed).blob())
    (t,) = [t for t in p["tasks"] if t["op"] == GEMM]
    assert [q["form"] for q in t["prob"]] == [0 if general or not FORMS[what] else FORMS[what] + (16 if dtype == "f16" else 0)]
    assert not [t for t in p["tasks"] if t["op"] not in (GEMM, FUSE_ROWS) and t["cut"]]


def test_epilogues_without_a_form_of_their_own(plan):
    """A 16-bit value that leaves as f32; 16-bit ones that are widened later do not."""
    for what, form in (("product", 0), ("residual", 3), ("gelu", 2), ("both", 3)):
        (t,) = [t for t in plan(progs.widened_product(256, 64, 256, "bf16", what).blob())["tasks"] if t["op"] == GEMM]
        assert [q["form"] for q in t["prob"]] == [form]


def test_few_rows_side_by_side_lie_spread_over_the_device(plan):
    """Tiles for 96 lanes of 148, two of three in use everywhere; on a kernel build that has the skinny products without the tiles of the
    tensor-core ones, which cost them registers."""
    p = plan(progs.products("bf16", *((16, 1024, 1024),) * 3).blob())
    lanes = sorted(lane for t in p["tasks"] for lane, _, _ in t["cut"])
    assert len(lanes) == len(set(lanes)) == 96 and all(0 < b - a <= 2 for a, b in zip(lanes, lanes[1:])) and lanes[0] == 0 and lanes[-1] >= 146
    builds = importlib.import_module("pjrt-ocl_b200.build").variants()
    gemm = int(re.search(r"kFamGemm = 1u << (\d+)", open(os.path.join(CSRC, "format.h")).read()).group(1))
    name, families = next((n, m) for n, m in builds if m & p["families"] == p["families"])
    assert name.startswith("plan") and not families >> gemm & 1
