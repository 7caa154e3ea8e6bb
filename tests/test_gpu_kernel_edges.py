"""The forms a call is dispatched to by its sizes, at the edges of each form: the one-pass short-sequence kernel (16-key
steps of its products, 32-column chunks, one and two 128-row tiles, its largest length and the one after it), the mask
ring of the tensor-core kernels (chunks of 32 keys; rows on 16-byte boundaries or not), the exact kernels' tiles and
key groups, and the 64-row steps of the tensor-core backward.  Every case against the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import (EXACT_FORWARD_SHAPES, TRAINING_SHAPES, TRAINING_SHAPES_LARGE, cosine, from_dev_bf16, max_abs,
                     normal_qkv, sawtooth_mask, to_dev, to_dev_bf16)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(attn_lib):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no fallback path to test")
    from autorust_b200 import ops as _ops
    return _ops


def _bf16(oracle_lib, arrays):
    return [oracle_lib.f32_to_bf16(x) for x in arrays]


def _assert_near_model(oracle_lib, got, model_mode, bits, mask, causal):
    """Against the oracle's model of the same rounding points.  Each side rounds P to bf16, possibly against another
    reference: 2^-9 of the weighted average of |v| each; the results are bf16, where a value next to a rounding boundary
    may fall on either side of it: 2^-7 of it; a quarter of the exponentials are within 1.1e-4, the others and the f32
    scores far inside that."""
    q, k, v = bits
    want = oracle_lib.bf16_to_f32(oracle_lib.flash(model_mode, q, k, v, mask, causal))
    size = oracle_lib.flash(0, *map(oracle_lib.bf16_to_f32, (q, k)), np.abs(oracle_lib.bf16_to_f32(v)), mask, causal)
    assert np.all(np.abs(got - want) <= 2.0 ** -7 * np.abs(want) + (2.0 ** -8 + 2.2e-4) * size)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 96, 127, 128, 129, 144, 160, 197, 255, 256, 257])
@pytest.mark.parametrize("causal", [False, True])
def test_bf16_short_sequences(ops, oracle_lib, n, causal):
    """The bf16 forward's 2e-2 against exact attention, and the model of its rounding points."""
    qb, kb, vb = _bf16(oracle_lib, normal_qkv(n, 2, 4, 2, n, 64))
    got = oracle_lib.bf16_to_f32(from_dev_bf16(ops.attn_forward("bf16", *map(to_dev_bf16, (qb, kb, vb)), None, causal)))
    exact = oracle_lib.flash(0, *map(oracle_lib.bf16_to_f32, (qb, kb, vb)), None, causal)
    assert max_abs(got, exact) <= 2e-2 and cosine(got, exact) >= 0.999
    _assert_near_model(oracle_lib, got, 2, (qb, kb, vb), None, causal)
    assert ops.last_status(None) == 0


def test_bf16_short_sequences_many_items_per_cta(ops, oracle_lib):
    """More (head, tile) items than resident CTAs: every CTA walks several, and its buffers change hands."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    B, H, S, D = 40, 12, 197, 64
    qkv = torch.randn(B, S, 3, H, D, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = (qkv[:, :, i].transpose(1, 2) for i in range(3))
    out = ops.attn_forward_views(q, k, v)
    want = torch.nn.functional.scaled_dot_product_attention(q.double(), k.double(), v.double())
    assert (out.double() - want).abs().max().item() <= 2e-2
    assert torch.equal(out, ops.attn_forward_views(q, k, v))
    # the last item alone gives the bits it had among the others
    one = ops.attn_forward_views(q[-1:], k[-1:], v[-1:])
    assert torch.equal(out[-1:], one)


@pytest.mark.parametrize("n", [1, 33, 100, 127, 128, 200, 256])
@pytest.mark.parametrize("causal", [False, True])
def test_short_log_sum_exp(ops, n, causal):
    """The row sums behind the training forward's log-sum-exp against float64 on the same bf16 operands.  Without a step
    of 128 visible keys every exponential is the MUFU unit's (2^-22) and the bound is that of f32 sums over values of a
    few units, 5e-6; a whole step has a quarter of its exponentials within 1.1e-4."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(2, 4, n, 64, device="cuda", generator=g) for _ in range(3))
    _, lse = ops.train_forward(q, k, v, causal=causal, tensor_cores=True)
    s = q.bfloat16().double() @ k.bfloat16().double().transpose(-1, -2) / 8.0
    if causal:
        s.masked_fill_(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    err = (lse.double() - torch.logsumexp(s, -1)).abs()
    whole = torch.arange(n, device="cuda") >= 128 if causal else torch.full((n,), n >= 128, device="cuda")
    assert err[..., ~whole].max().item() <= 5e-6 if (~whole).any() else True
    assert err[..., whole].max().item() <= 3.5e-5 if whole.any() else True


@pytest.mark.parametrize("n", [40, 128, 129, 200, 256])
def test_short_and_long_kernel_give_a_row_the_same_bits(ops, n):
    """A causal row sees the same keys in a call of n tokens (the one-pass kernel) and in one of 300 (the key loop): the
    same steps, references and sums."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(1, 3, 300, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    long = ops.attn_forward("bf16", q, k, v, None, True)
    short = ops.attn_forward("bf16", *(t[:, :, :n].contiguous() for t in (q, k, v)), None, True)
    assert torch.equal(short, long[:, :, :n])


@pytest.mark.parametrize("mode,d", [("bf16", 64), ("bf16", 128), ("tf32", 64), ("sage_fp8", 64), ("sage_fp8", 128), ("sage", 128),
                                    ("sage_rows", 64)])
@pytest.mark.parametrize("n", [1, 31, 33, 100, 127, 129, 260, 389])
@pytest.mark.parametrize("causal", [False, True])
def test_mask_ring(ops, oracle_lib, mode, d, n, causal):
    """An additive mask of N(0,1) values with masked-out (-1e30) columns, its rows on 16-byte boundaries (n a multiple
    of 4) or not, one and two query tiles per CTA (bf16 D = 64 up to 128 tokens); the modes' own bounds against exact
    attention with that mask, or the model of their rounding points.  (The INT8 modes read their mask in place.)"""
    import torch
    q, k, v = normal_qkv(n, 1, 2, 1, n, d)
    mask = np.random.default_rng(n).standard_normal((n, n)).astype(np.float32)
    mask[:, n - n // 4:] = -1e30
    if mode == "tf32":
        dev, exact = [to_dev(x) for x in (q, k, v)], oracle_lib.flash(0, q, k, v, mask, causal)
    else:
        bits = _bf16(oracle_lib, (q, k, v))
        dev, exact = [to_dev_bf16(x) for x in bits], oracle_lib.flash(0, *map(oracle_lib.bf16_to_f32, bits), mask, causal)
    out = ops.attn_forward(mode, *dev, to_dev(mask), causal)
    got = out.float().cpu().numpy()
    # the quantised modes: a row of few visible keys carries the INT8 rounding of single logits
    if mode == "sage_fp8":
        _assert_near_model(oracle_lib, got, 4, bits, mask, causal)
    else:
        bound = {"bf16": 2e-2, "tf32": 5e-3, "sage": 1e-1, "sage_rows": 1e-1}[mode]
        assert max_abs(got, exact) <= bound and cosine(got, exact) >= 0.999
    # the same values at an address that is 4-byte but not 16-byte aligned take the other copy width: the same bits
    shifted = torch.cat([torch.zeros(1), torch.from_numpy(mask).flatten()]).cuda()[1:].view(n, n)
    assert torch.equal(out, ops.attn_forward(mode, *dev, shifted, causal))
    assert ops.last_status(None) == 0


@pytest.mark.parametrize("b,hq,hkv,n", EXACT_FORWARD_SHAPES)
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_exact_tiles(ops, oracle_lib, b, hq, hkv, n, d, causal):
    """Every form of the tile rule (tests/test_plans.py), the key groups with more groups than tiles, with a mask at some
    lengths; 1e-5 of the largest value as for the exact mode elsewhere."""
    q, k, v = normal_qkv(n, b, hq, hkv, n, d)
    mask = sawtooth_mask(n) if n in (17, 50, 65, 197, 257) else None
    got = ops.attn_forward("exact", *map(to_dev, (q, k, v)), None if mask is None else to_dev(mask), causal).cpu().numpy()
    want = oracle_lib.flash(0, q, k, v, mask, causal)
    assert np.all(np.abs(got - want) <= 1e-5 * np.maximum(np.abs(want), 1.0))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n", [40, 100, 200, 330])
def test_exact_causal_rows_without_visible_keys(ops, n, d):
    """Left padding under a causal mask: a row whose visible keys all carry -1e30 averages V over the keys up to the end of
    the 64 its diagonal lies in (those past the sequence end count as zeros), in every batch and head and whatever
    tile height B * H * S selects.  Other rows are the attention over their visible keys."""
    import torch
    pad = n - n // 3
    mask = torch.zeros(n, n, device="cuda")
    mask[:, :pad] = -1e30
    g = torch.Generator(device="cuda").manual_seed(n)
    q1, k1, v1 = (torch.randn(1, 1, n, d, device="cuda", generator=g) for _ in range(3))
    s = q1[0, 0].double() @ k1[0, 0].double().T / d ** 0.5 + mask.double()
    s.masked_fill_(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.softmax(s, -1) @ v1[0, 0].double()
    for row in range(pad):
        end = (row // 64 + 1) * 64
        want[row] = v1[0, 0, :end].double().sum(0) / end
    for heads in (1, 6, 24, 60, 148, 400):
        q, k, v = (t.expand(1, heads, n, d).contiguous() for t in (q1, k1, v1))
        got = ops.attn_forward("exact", q, k, v, mask, True)
        # the outputs are averages of N(0,1) values, below about 5: the exact mode's 1e-5 of the largest value
        assert (got[0].double() - want).abs().max().item() <= 1e-5, heads


@pytest.mark.parametrize("tc", [False, True])
@pytest.mark.parametrize("b,hq,hkv,n", TRAINING_SHAPES)
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_training_steps(ops, oracle_lib, tc, b, hq, hkv, n, d, causal):
    """Every form of both backwards without a causal mask (tests/test_plans.py), fewer steps than stages, ragged tiles,
    several query heads per K/V head, with and without a mask.  Exact: 2e-5 of
    the largest entry, as the training tests hold it.  bf16 operands: 2e-2 of it (dP is a sum of D products of operands
    rounded to 2^-9, off by 2^-9 sqrt(2 D / 3) = 0.018 in the root mean square at D = 128, and a row of few visible keys
    passes that on to its dQ undamped), and a cosine of 0.9995."""
    import torch
    rng = np.random.default_rng(n)
    q, k, v = normal_qkv(n, b, hq, hkv, n, d)
    d_o = rng.standard_normal(q.shape, dtype=np.float32)
    mask = sawtooth_mask(n) if n in (65, 127, 129) else None
    want = dict(zip(("o", "lse", "dq", "dk", "dv"), oracle_lib.attn_train(q, k, v, d_o, mask, causal)))
    tq, tk, tv, tdo = map(to_dev, (q, k, v, d_o))
    tm = None if mask is None else to_dev(mask)
    o, lse = ops.train_forward(tq, tk, tv, tm, causal, tensor_cores=tc)
    grads = ops.train_backward(tq, tk, tv, o, tdo, lse, tm, causal, tensor_cores=tc)
    again = ops.train_backward(tq, tk, tv, o, tdo, lse, tm, causal, tensor_cores=tc)
    for name, got in zip(("o", "lse", "dq", "dk", "dv"), (o, lse, *grads)):
        w = want[name]
        bound = (2e-2 if tc else 2e-5) * max(1.0, float(np.abs(w).max()))
        assert max_abs(got.cpu().numpy(), w) <= bound, (name, max_abs(got.cpu().numpy(), w), bound)
        if np.abs(w).max() > 1e-3:  # (one key: dQ and dK are zero)
            assert cosine(got.cpu().numpy(), w) >= 0.9995, name
    for x, y in zip(grads, again):  # no atomics: two launches give the same bits
        assert torch.equal(x, y)
    assert ops.last_status(None) == 0


@pytest.mark.parametrize("tc", [False, True])
@pytest.mark.parametrize("b,hq,hkv,n", TRAINING_SHAPES_LARGE)
@pytest.mark.parametrize("masked", [False, True])
def test_training_steps_of_many_causal_heads(ops, tc, b, hq, hkv, n, masked):
    """The forms that only large causal calls take (128-row exact tiles, two tensor-core CTAs per SM), against float64
    autograd on the GPU; the bounds of test_training_steps."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, d_o = (torch.randn(b, h, n, 64, device="cuda", generator=g) for h in (hq, hkv, hkv, hq))
    mask = torch.randn(n, n, device="cuda", generator=g) if masked else None
    o, lse = ops.train_forward(q, k, v, mask, True, tensor_cores=tc)
    got = ops.train_backward(q, k, v, o, d_o, lse, mask, True, tensor_cores=tc)
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) / 8.0
    if masked:
        s = s + mask.double()
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    (torch.softmax(s, -1) @ vd).backward(d_o.double())
    for name, x, w in zip(("dq", "dk", "dv"), got, (qd.grad, kd.grad, vd.grad)):
        bound = (2e-2 if tc else 2e-5) * max(1.0, w.abs().max().item())
        assert (x.double() - w).abs().max().item() <= bound, name
        assert torch.nn.functional.cosine_similarity(x.double().flatten(), w.flatten(), dim=0).item() >= 0.9995, name
    assert ops.last_status(None) == 0


@pytest.mark.parametrize("mode,b,hq,hkv,n", [("bf16", 1, 16, 16, 8200), ("sage", 1, 32, 32, 4100), ("sage_fp8", 1, 32, 32, 5000)])
def test_heads_in_several_groups(ops, mode, b, hq, hkv, n):
    """K and V of more heads than are walked together (32 MB), and a partial last tile: a grid of several groups.  Each head
    alone, in a plain grid, gives the same bits; bf16 through strided views as well."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(b, h, n, 128, device="cuda", generator=g).to(torch.bfloat16) for h in (hq, hkv, hkv))
    for causal in (False, True):
        out = ops.attn_forward(mode, q, k, v, None, causal)
        for h in (0, 1, hq // 2, hq - 1):
            kv = h // (hq // hkv)
            one = ops.attn_forward(mode, q[:, h:h + 1].contiguous(), *(t[:, kv:kv + 1].contiguous() for t in (k, v)), None, causal)
            assert torch.equal(out[:, h:h + 1], one), (causal, h)
        if mode == "bf16":
            views = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)]
            assert torch.equal(out, ops.attn_forward_views(*views, None, causal))
    assert ops.last_status(None) == 0


@pytest.mark.parametrize("n,d", [(200, 64), (700, 128)])
def test_captured_call_between_ticketed_ones(ops, n, d):
    """Calls outside of a capture mark the shared status word with a ticket, a captured one clears it: replays between
    such calls give the bits of the eager call and leave nothing behind."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn(2, 80, n, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    want = ops.attn_forward("bf16", q, k, v)
    out = torch.empty_like(q)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ops.attn_forward("bf16", q, k, v, out=out)
    for _ in range(3):
        out.zero_()
        assert torch.equal(ops.attn_forward("bf16", q, k, v), want)
        graph.replay()
        assert torch.equal(ops.attn_forward("bf16", q, k, v), want)
        assert torch.equal(out, want)
    assert ops.last_status(None) == 0
