"""Which decode kernel `kernels.linear` hands a bfloat16 product to (no GPU needed: the rule only looks at sizes)."""
import ast
import glob
import inspect
import os

import pytest
import torch

from tq_kv_b200.kernels import gemm, scan


def _w(n, k):
    return torch.empty(n, k, dtype=torch.bfloat16, device="meta")


@pytest.mark.parametrize("rows,n,k,swiglu,after_norm,f32,want", [
    # the 7B shape: everything on the tcgen05 kernel
    (8, 4608, 3584, False, True, True, True),
    (8, 3584, 3584, False, False, True, True),
    (8, 2 * 18944, 3584, True, True, False, True),
    (8, 3584, 18944, False, False, True, True),
    # the 0.5B shape at 8 rows: q|k|v (norm folded in), o and gate|up stay on the mma.sync kernel, down does not
    (8, 1152, 896, False, True, True, False),
    (8, 896, 896, False, False, True, False),
    (8, 2 * 4864, 896, True, True, False, False),
    (8, 896, 4864, False, False, True, True),
    # from 9 rows on the float32 results of given rows leave the mma.sync kernel at any size
    (9, 896, 896, False, False, True, True),
    (9, 1152, 896, False, True, True, False),
    # a 55 MB gated product stays, a 90 MB one does not
    (8, 2 * 8960, 1536, True, True, False, False),
    (8, 2 * 11008, 2048, True, True, False, True),
    # from 9 rows on gated products leave it from 40 MB
    (9, 2 * 4864, 896, True, True, False, False),
    (16, 2 * 8192, 1024, True, True, False, False),
    (9, 2 * 10240, 1024, True, True, False, True),
    (16, 2 * 5632, 2048, True, True, False, True),
    # over 16 rows, or with K no multiple of 32, only the tcgen05 kernel can
    (17, 896, 896, False, False, True, True),
    (4, 64, 40, False, False, True, True),
])
def test_which_decode_kernel_takes_a_product(rows, n, k, swiglu, after_norm, f32, want):
    assert gemm._tc_takes(rows, _w(n, k), swiglu, after_norm, f32) is want


@pytest.mark.parametrize("rows, n, k, swiglu, want", [
    (1, 1152, 896, False, False), (1, 10304, 2048, False, True), (2, 10304, 2048, False, False),
    (1, 2 * 5632, 2048, True, True), (1, 2 * 4864, 896, True, False), (1, 2 * 18944, 3584, True, False),
    (1, 896, 4864, False, False), (1, 2048, 5632, False, True), (1, 3584, 18944, False, False),
    (1, 151936, 896, False, True), (1, 152064, 3584, False, True), (2, 151936, 896, False, False)])
def test_which_products_of_one_row_run_on_the_row_kernel(rows, n, k, swiglu, want):
    assert gemm._row_takes(rows, _w(n, k), swiglu) is want


def test_parts_say_that_their_weights_are_settled_and_nobody_else_is_taken_to():
    """A product reads a settled weight before the kernel in front has ended: true of a model's weights, not of any w."""
    assert inspect.signature(gemm.linear).parameters["w_settled"].default is False
    calls = 0
    for path in sorted(glob.glob(os.path.join(os.path.dirname(gemm.__file__), "..", "parts", "*.py"))):
        with open(path) as f:
            for node in ast.walk(ast.parse(f.read())):
                if isinstance(node, ast.Call) and isinstance(node.func, ast.Attribute) and node.func.attr == "linear":
                    calls += 1
                    said = {k.arg: getattr(k.value, "value", None) for k in node.keywords}
                    assert said.get("w_settled") is True, (path, node.lineno)
                    assert isinstance(node.args[1], ast.Attribute), (path, node.lineno)        # self.w_..., a weight
    assert calls > 30


@pytest.mark.parametrize("rows, n, want", [(8, 5_000_000, True), (9, 64 * 65535, True), (9, 64 * 65535 + 1, False), (300, 5_000_000, False)])
def test_float32_products_with_more_columns_than_a_grid_has_tiles_for(rows, n, want):
    x, w, out = (torch.empty(s, device="meta") for s in ((rows, 4), (n, 4), (rows, n)))
    assert gemm._f32_ok(x, w, out) is want


@pytest.mark.parametrize("mode, silu, tokens, seqs, width, want", [
    (scan.SCAN_DELTA, False, 8, 1, 256, True), (scan.SCAN_DELTA, False, 15, 1, 128, False), (scan.SCAN_DELTA, False, 16, 1, 128, True),
    (scan.SCAN_DELTA, False, 47, 1, 64, False), (scan.SCAN_DELTA, False, 191, 1, 32, False), (scan.SCAN_DELTA, False, 192, 1, 32, True),
    (scan.SCAN_DECAY, True, 31, 1, 128, False), (scan.SCAN_DECAY, True, 64, 2, 128, True), (scan.SCAN_DECAY, False, 40, 1, 128, False),
    (scan.SCAN_GATED, False, 3000, 1, 128, True), (scan.SCAN_GATED, False, 90, 2, 128, False), (scan.SCAN_GATED, False, 90, 1, 32, False),
    (scan.SCAN_GATED_DELTA, False, 48, 1, 64, True), (scan.SCAN_GATED_DELTA, False, 200, 1, 32, False)])
def test_how_long_a_step_goes_eight_tokens_at_a_time(mode, silu, tokens, seqs, width, want):
    assert scan._long_enough(mode, silu, tokens, seqs, width) is want


@pytest.mark.parametrize("use", [True, False])
def test_the_tcgen05_switch_leaves_the_row_kernel_alone(use, monkeypatch):
    """It runs on FMA units."""
    monkeypatch.setattr(gemm, "USE_TCGEN05", use)
    ran = []
    monkeypatch.setattr(gemm, "row_gemm", lambda x, w, out, *a: ran.append(w.shape) or out)
    gemm.linear(torch.empty(1, 2048, dtype=torch.bfloat16, device="meta"), _w(10304, 2048))
    assert ran == [(10304, 2048)]
