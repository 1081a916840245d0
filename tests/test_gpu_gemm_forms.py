"""Every form of the uint8 tensor-core GEMM against exact integer arithmetic, all rows bit for bit.

The launcher picks single CTAs or pairs, a tile height, K slices and the chunks per ring stage from the sizes; the
cases below reach all of them on 148 SMs, with partial last row tiles, partial last weight tiles, an odd number of
chunks per tile or slice where a stage takes two, and several tiles per CTA where the accumulator has one buffer."""
import pytest
import torch

from rwkvstic_b200 import _lib

from kernel_contract import QMAX

DEV = "cuda:0"
SMS = 148

# (pair, activation rows per CTA, K slices, chunks per stage): (rows, outputs of each matrix, inputs)
FORMS = {
    (0, 16, 1, 1): (5, [129], 128),
    (0, 16, 1, 2): (13, [129], 384),
    (0, 16, 2, 2): (7, [129], 3328),
    (0, 16, 4, 2): (9, [300], 2560),
    (0, 16, 8, 2): (15, [129], 5120),
    (0, 32, 1, 1): (36, [5952, 3329], 128),
    (0, 32, 1, 2): (1208, [257], 384),
    (0, 32, 2, 2): (17, [4737], 4864),
    (0, 32, 4, 2): (293, [131], 2560),
    (0, 32, 8, 2): (17, [1153], 5120),
    (0, 48, 1, 1): (35, [14209, 13888, 9475], 1280),
    (0, 64, 1, 1): (197, [5633, 5123, 3200], 128),
    (0, 80, 1, 1): (196, [1409, 6785, 5952], 128),
    (1, 16, 1, 2): (17, [131, 8707, 513], 1152),
    (1, 32, 1, 1): (33, [1281, 8067], 1792),
    (1, 48, 1, 1): (82, [8707, 13441, 6147], 1792),
    (1, 64, 1, 1): (332, [6915, 4736, 3840], 3200),
    (1, 80, 1, 1): (595, [5184, 7681], 1152),
}


@pytest.mark.parametrize("form", FORMS, ids=str)
def test_the_case_has_the_form_it_stands_for(form):
    rows, n_out, k = FORMS[form]
    plan = _lib.gemm_plan(1, k, n_out, rows, SMS)
    assert (plan["pair"], plan["rows"], plan["slices"], plan["chunks"]) == form
    if plan["buffers"] == 1:        # the single buffer is handed over more than once
        row_tiles = -(-rows // (plan["rows"] * (1 + plan["pair"])))
        assert row_tiles * sum(-(-n // 256) for n in n_out) > SMS // 2


def test_every_tile_height_is_covered():
    assert {(f[0], f[1]) for f in FORMS} == {(p, r) for p in (0, 1) for r in (16, 32, 48, 64, 80)}
    assert {f[2] for f in FORMS} == {1, 2, 4, 8}


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS, ids=str)
def test_integer_sums_of_every_row_are_exact(form):
    from test_gpu_kernels import random_matrix
    from test_gpu_rows import run_gemm
    rows, n_out, k = FORMS[form]
    g = torch.Generator().manual_seed(rows + k)
    mats = [random_matrix(n, k, seed=n + k, zero_offset=True) for n in n_out]
    xs = [torch.randn(rows, k, generator=g) * 3 for _ in mats]
    for x in xs:
        x[rows // 2] *= 1e-3                       # scaling is per row
    first = run_gemm(mats, xs)
    for m, x, got in zip(mats, xs, first):
        s = x * m.ry
        inv = torch.tensor(QMAX) / s.abs().amax(dim=1, keepdim=True)
        X = torch.round(s * inv).double().to(DEV)                     # whole numbers below 2^23
        total = X @ m.qt.to(DEV).double().t()                         # exact: below 2^44
        want = total.to(torch.float32).cpu() * (1.0 / inv)
        assert torch.equal(got, want)
    again = run_gemm(mats, xs)                     # the scratch of K slices is left as it was found
    assert all(torch.equal(a, b) for a, b in zip(first, again))


@pytest.mark.parametrize("rows,n_out,k", [(773, [2048], 256), (512, [768] * 3, 768), (39, [3072] * 3, 128), (73, [4096] * 2, 128)])
def test_a_short_sum_takes_tiles_that_its_epilogue_does_not_bound(rows, n_out, k):
    """With few steps of K a tile costs its epilogue, and pair tiles cost more of it a row than single ones need: these
    sizes ran 6 to 20 % slower in pair tiles of 32 and 64 rows than in the form they take."""
    plan = _lib.gemm_plan(1, k, n_out, rows, SMS)
    assert (plan["pair"], 2 * plan["rows"]) not in {(1, 32), (1, 64)}
