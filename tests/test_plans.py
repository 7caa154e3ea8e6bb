"""The forms that calls are dispatched to by their sizes (ar_attn_plan; no GPU needed): launches stay inside the grid's limits
over the sizes that the entry points accept, and the rules give the forms that were measured ahead."""
from __future__ import annotations

import pytest

from autorust_b200 import _abi


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
