"""The forms that calls are dispatched to by their sizes (ar_attn_plan; no GPU needed): launches stay inside the grid's limits
over the sizes that the entry points accept, and the rules give the forms that were measured ahead."""
from __future__ import annotations

import pytest

from autorust_b200 import _abi
from helpers import EXACT_FORWARD_SHAPES, TRAINING_SHAPES, TRAINING_SHAPES_LARGE


@pytest.fixture(scope="module", autouse=True)
def _lib(attn_lib):
    return attn_lib


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("s", [1, 64, 4194240, 4194241, 1 << 24])
@pytest.mark.parametrize("b,hq,hkv", [(1, 1, 1), (1, 8, 2), (5, 60, 60), (1, 65535, 65535)])
def test_exact_backward_grids_fit(b, hq, hkv, s, causal, d):
    dq_rows, dkv_rows, *grids = _abi.plan(_abi.PLAN_TRAIN_BACKWARD, b, hq, hkv, s, d, causal)
    for rows, heads, (x, y, z) in ((dq_rows, b * hq, grids[:3]), (dkv_rows, b * hkv, grids[3:])):
        assert 1 <= y <= 65535 and 1 <= z <= 65535 and 1 <= x < 1 << 31
        assert x * y * z == -(-s // rows) * heads


@pytest.mark.parametrize("causal", [False, True])
def test_tc_backward_forms(causal):
    """Two CTAs per SM for many short walks at D = 64, one CTA per SM elsewhere; a cluster per GQA group only where the key
    tiles alone would leave SMs idle over long walks."""
    plan = lambda *sizes: _abi.plan(_abi.PLAN_TRAIN_BACKWARD_TC, *sizes, causal)[:3]
    assert plan(1, 768, 768, 64, 64) == [1, 1, 1]
    assert plan(1, 768, 768, 197, 64) == [1, 1, 1]
    assert plan(1, 768, 768, 197, 128) == [0, 0, 1]
    assert plan(1, 24, 24, 768, 64) == [0, 0, 1]      # 144 CTAs: one round
    assert plan(1, 1, 1, 1, 64) == [0, 0, 1]
    assert plan(1, 16, 2, 1531, 64)[2] >= 4           # 24 key tiles, 8 query heads each
    assert plan(1, 16, 2, 1531, 128)[2] >= 4
    for b, hq, hkv, s, d in ((36, 64, 8, 256, 64), (16, 64, 8, 512, 64), (8, 56, 8, 1000, 64), (16, 40, 8, 384, 128),
                             (36, 16, 8, 197, 128), (8, 64, 8, 197, 64)):
        assert plan(b, hq, hkv, s, d)[2] == 1
    group = plan(3, 21, 3, 500, 64)[2]
    assert 7 % group == 0


def test_grids_are_grouped_only_where_tiles_differ():
    """Heaviest tiles first for the heads of a group: under a causal mask or with a partial tile.  Tiles of one weight keep
    the grid of (tiles, heads), whose CTAs side by side share few heads' K and V."""
    grid = lambda *sizes: tuple(_abi.plan(_abi.PLAN_TRAIN_BACKWARD, *sizes)[2:5])
    assert grid(1, 148, 148, 256, 64, False) == (2, 148, 1)
    heads_of_a_group, tiles, groups = grid(1, 148, 148, 250, 64, False)
    assert (heads_of_a_group * groups, tiles) == (148, 2) and heads_of_a_group > 1
    heads_of_a_group, tiles, groups = grid(1, 20, 20, 512, 64, True)
    assert (heads_of_a_group * groups, tiles) == (20, 8) and heads_of_a_group > 1


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("d,forms", [(64, {8, 12, 16, 20, 24, 32, 64, 128}), (128, {8, 12, 16, 20, 24, 32, 64})])
def test_the_numerics_tests_reach_every_form_of_the_exact_forward(d, forms, causal):
    plans = [_abi.plan(_abi.PLAN_EXACT_FORWARD, b, hq, hkv, n, d, causal)[:2] for b, hq, hkv, n in EXACT_FORWARD_SHAPES]
    assert {rows for rows, plain in plans if not plain} == forms
    assert [64, 1] in plans


def test_the_numerics_tests_reach_every_form_of_the_backwards():
    exact = lambda shapes, causal: {tuple(_abi.plan(_abi.PLAN_TRAIN_BACKWARD, *s, 64, causal)[:2]) for s in shapes}
    assert exact(TRAINING_SHAPES, False) == {(64, 64), (64, 128), (128, 64), (128, 128)}
    assert (128, 128) in exact(TRAINING_SHAPES_LARGE, True) and (64, 64) in exact(TRAINING_SHAPES, True)
    for causal in (False, True):
        fast = [_abi.plan(_abi.PLAN_TRAIN_BACKWARD_TC, *s, 64, causal)[:3] for s in TRAINING_SHAPES + TRAINING_SHAPES_LARGE]
        assert [0, 0, 1] in fast and [1, 1, 1] in fast and any(split > 1 for _, _, split in fast)
        fast = [_abi.plan(_abi.PLAN_TRAIN_BACKWARD_TC, *s, 128, causal)[:3] for s in TRAINING_SHAPES]
        assert [0, 0, 1] in fast and any(split > 1 for _, _, split in fast)


def test_exact_forward_form_of_many_short_and_many_long_heads():
    """The forms that were measured ahead: the plain one for many heads of one key tile (48 heads of S=50, causal: 8.6 us
    against 14.2 with 12-row tiles), 128-row tiles for large calls, tiles of 16 to 24 rows for one image's layer."""
    form = lambda *sizes: _abi.plan(_abi.PLAN_EXACT_FORWARD, *sizes)[:2]
    for d in (64, 128):
        assert form(1, 200, 200, 50, d, True) == [64, 1]
    assert form(8, 32, 32, 2048, 64, False) == [128, 0]
    assert form(16, 16, 16, 188, 128, False) == [64, 0]   # 174 us; the plain one 217
    assert form(1, 12, 12, 197, 64, False)[0] in (16, 20, 24)


def test_exact_backward_forms_of_causal_calls():
    """Under a causal mask the 128-row kernels want more than four rounds of CTAs (200 heads of S=197: 297 us against 229
    with 64 rows; 96 heads of S=848: 1110 against 1230)."""
    rows = lambda *sizes: _abi.plan(_abi.PLAN_TRAIN_BACKWARD, *sizes, 64, True)[:2]
    for heads, n in ((200, 197), (200, 256), (200, 300), (96, 500), (96, 700), (48, 848), (352, 405)):
        assert rows(1, heads, heads, n) == [64, 64]
    for heads, n in ((96, 848), (200, 500), (200, 512)):
        assert rows(1, heads, heads, n) == [128, 128]
