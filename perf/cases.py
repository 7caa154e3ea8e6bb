"""The work a user of this package has it do, as timed cases: the attention forward in each of its modes, the training
step, and the ViT-B/16 encoder around the operator.

`listed()` are the cases timed by name, `draw(rng)` gives more of the same ranges.  `prepare` makes what a program holds
before the call (tensors on the GPU, a model), `run` is one pass through the public entry points of autorust_b200.ops and
autorust_b200.vit, `work` the bytes and operations a pass cannot do without, `tolerance` how far another correct
implementation at the same precision may be from this one.
"""
import torch

from autorust_b200 import ops
from autorust_b200.vit import ViT

# The most operations a drawn case of a kind may have: at most about the time of the largest listed case (the exact mode
# works at f32 precision, the tensor-core modes at bf16 or 8 bits).
MOST_FLOPS = {"exact": 4e10, "tf32": 2e11, "bf16": 1e12, "sage": 1e12, "sage_fp8": 1e12, "train_exact": 3e10, "train_tc": 4e11}
IMAGE, PATCH, EMBED, HEADS, LAYERS, CLASSES = 224, 16, 768, 12, 12, 1000


def _attn(name, mode, B, Hq, Hkv, S, D, causal=False, mask=False, views=False):
    return {"name": name, "kind": "forward", "mode": mode, "B": B, "Hq": Hq, "Hkv": Hkv, "S": S, "D": D, "causal": causal,
            "mask": mask, "views": views}


def _train(name, tensor_cores, B, Hq, Hkv, S, D, causal=False):
    return {"name": name, "kind": "train", "tensor_cores": tensor_cores, "B": B, "Hq": Hq, "Hkv": Hkv, "S": S, "D": D,
            "causal": causal}


def listed():
    return [
        # one image through one layer's attention in full precision: the smallest call, mostly latency
        _attn("exact_vit_layer", "exact", 1, 12, 12, 197, 64),
        # f32 tensors in the fast mode, a small vision transformer's batch (odd length)
        _attn("tf32_s789", "tf32", 8, 6, 6, 789, 64),
        # a padded batch with a position bias: the additive [S, S] mask
        _attn("bf16_masked", "bf16", 4, 16, 16, 789, 64, mask=True),
        # the ViT-B/16 layer at batch 64: q, k, v are slices of one fused projection, read in place
        _attn("bf16_vit_views", "bf16", 64, 12, 12, 197, 64, views=True),
        # language-model prefill
        _attn("bf16_causal_prefill", "bf16", 8, 32, 32, 4096, 128, causal=True),
        # grouped-query prefill of a ragged prompt with quantised Q and K
        _attn("sage_gqa_prefill", "sage", 2, 32, 8, 3001, 128, causal=True),
        # the benchmark's workload: long non-causal INT8 attention
        _attn("sage_long", "sage", 4, 32, 32, 8192, 128),
        # training step, forward and backward, in full precision (what the host API's training calls run)
        _train("train_exact", False, 2, 8, 8, 1024, 64),
        # training step in the fast mode
        _train("train_fast", True, 4, 16, 16, 2048, 64),
        # the same for a causal model with grouped heads and an odd length
        _train("train_fast_gqa", True, 2, 16, 4, 1531, 128, causal=True),
        # one image and one batch through the whole encoder
        {"name": "vit_b1", "kind": "vit", "batch": 1},
        {"name": "vit_b64", "kind": "vit", "batch": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["forward"] * 6 + ["train"] * 3 + ["vit"])
    if kind == "vit":
        return {"kind": "vit", "batch": _log_int(rng, 1, 64)}
    if kind == "train":
        tc = rng.random() < 0.6
        which = "train_tc" if tc else "train_exact"
    else:
        which = rng.choice(["exact", "tf32", "bf16", "bf16", "bf16", "sage", "sage", "sage_fp8"])
    D = 64 if which == "tf32" else rng.choice([64, 128])
    causal = rng.random() < 0.5
    while True:
        S = _log_int(rng, 50, 8192)
        B = _log_int(rng, 1, 32)
        Hkv = rng.choice([1, 2, 4, 6, 8, 12, 16, 32])
        Hq = Hkv * rng.choice([1, 1, 1, 2, 4])
        case = {"B": B, "Hq": Hq, "Hkv": Hkv, "S": S, "D": D, "causal": causal}
        if kind == "train":
            case.update(kind="train", tensor_cores=tc)
        else:
            mask = S <= 2048 and rng.random() < 0.2
            case.update(kind="forward", mode=which, mask=mask, views=which == "bf16" and Hq == Hkv and rng.random() < 0.3)
        w = work(case)
        if w["flops"] <= MOST_FLOPS[which] and w["bytes"] <= 1e9:
            return case


def _normal(gen, *shape, dtype=torch.float32):
    return torch.randn(shape, device="cuda", generator=gen).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "vit":
        images = torch.rand(case["batch"], 3, IMAGE, IMAGE, device="cuda", generator=gen)
        return {"kind": "vit", "model": ViT(layers=LAYERS, embed_dim=EMBED, num_heads=HEADS, img_size=IMAGE, patch_size=PATCH,
                                            num_classes=CLASSES, seed=seed), "images": images}
    B, Hq, Hkv, S, D = (case[k] for k in ("B", "Hq", "Hkv", "S", "D"))
    if case["kind"] == "train":
        return {"kind": "train", "tensor_cores": case["tensor_cores"], "causal": case["causal"], "q": _normal(gen, B, Hq, S, D),
                "k": _normal(gen, B, Hkv, S, D), "v": _normal(gen, B, Hkv, S, D), "d_o": _normal(gen, B, Hq, S, D)}
    mode = case["mode"]
    dtype = torch.float32 if mode in ("exact", "tf32") else torch.bfloat16
    state = {"kind": "forward", "mode": mode, "views": case["views"], "causal": case["causal"], "mask": None}
    if case["views"]:  # slices of one [B, S, 3 * H * D] projection
        qkv = _normal(gen, B, S, 3, Hq, D, dtype=dtype)
        state.update((name, qkv[:, :, i].transpose(1, 2)) for i, name in enumerate(("q", "k", "v")))
    else:
        # the quantised modes meet a K with a large offset per channel; that is what their smoothing is for
        offset = 2.0 * _normal(gen, 1, Hkv, 1, D) if mode.startswith("sage") else 0.0
        state["q"] = _normal(gen, B, Hq, S, D, dtype=dtype)
        state["k"] = (_normal(gen, B, Hkv, S, D) + offset).to(dtype)
        state["v"] = _normal(gen, B, Hkv, S, D, dtype=dtype)
    if case["mask"]:  # a bias that falls off with the distance; the last keys are padding
        at = torch.arange(S, device="cuda", dtype=torch.float32)
        slope = 0.01 * (1.0 + float(torch.rand((), generator=gen, device="cuda")))
        mask = -slope * (at[:, None] - at[None, :]).abs()
        mask[:, S - S // 10:] = -1e30
        state["mask"] = mask.contiguous()
    return state


def run(state):
    if state["kind"] == "vit":
        return state["model"].forward(state["images"])
    q, k, v = state["q"], state["k"], state["v"]
    if state["kind"] == "train":
        tc, causal = state["tensor_cores"], state["causal"]
        o, lse = ops.train_forward(q, k, v, causal=causal, tensor_cores=tc)
        dq, dk, dv = ops.train_backward(q, k, v, o, state["d_o"], lse, causal=causal, tensor_cores=tc)
        return {"o": o, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    if state["views"]:
        return ops.attn_forward_views(q, k, v, state["mask"], state["causal"])
    return ops.attn_forward(state["mode"], q, k, v, state["mask"], state["causal"])


def work(case):
    if case["kind"] == "vit":
        n, e = case["batch"], EMBED
        patches = (IMAGE // PATCH) ** 2
        s = patches + 1
        layer = 2 * s * e * 12 * e + 4 * s * s * e  # four projections of E x E, the MLP of 2 x E x 4E, the attention
        flops = n * (2 * patches * e * 3 * PATCH * PATCH + LAYERS * layer + 2 * e * CLASSES)
        weights = e * 3 * PATCH * PATCH + s * e + LAYERS * 12 * e * e + e * CLASSES
        return {"bytes": 2 * weights + n * (4 * 3 * IMAGE * IMAGE + 2 * CLASSES), "flops": flops}
    B, Hq, Hkv, S, D = (case[k] for k in ("B", "Hq", "Hkv", "S", "D"))
    pairs = S * (S + 1) // 2 if case["causal"] else S * S
    product = 2 * B * Hq * pairs * D
    q_elems, kv_elems = B * Hq * S * D, B * Hkv * S * D
    if case["kind"] == "train":  # in: q, k, v, dO; out: o, lse, dq, dk, dv; two products forward, five backward
        return {"bytes": 4 * (4 * q_elems + 4 * kv_elems + B * Hq * S), "flops": 7 * product}
    size = 4 if case["mode"] in ("exact", "tf32") else 2
    return {"bytes": size * 2 * (q_elems + kv_elems) + (4 * S * S if case["mask"] else 0), "flops": 2 * product}


def tolerance(case):
    # About four times the distance to the same computation in 64 bits (the quantised modes: on the same 8-bit tensors),
    # measured over the listed and a dozen drawn cases: relative error at most 7.2e-7 exact (S = 1024; it grows with the
    # root of S), 1.7e-3 TF32, 2.4e-3 for the bf16 P of the forward modes, 4.3e-3 for the bf16 P and dS of the fast
    # gradients, 1.2e-2 through the encoder's twelve bf16 layers (there the largest value that may be stated counts).
    if case["kind"] == "vit":
        return {"rel": 0.03, "max": 0.2}
    if case["kind"] == "train":
        return {"rel": 0.017, "max": 0.5} if case["tensor_cores"] else {"rel": 8e-6, "max": 8e-5}
    if case["mode"] == "exact":
        return {"rel": 8e-6, "max": 8e-5}
    return {"rel": 6.5e-3, "max": 0.05} if case["mode"] == "tf32" else {"rel": 0.01, "max": 0.17}
