"""What a user of the attention library has it do, as cases that can be timed and compared.

``listed()`` gives the representative calls, ``draw(rng)`` more of the same ranges.  Every case is one pass
through a public entry point: the ``MonarchAttention`` module on device tensors (``"call": "module"``), the
module under autograd (``"train"``), or ``monarch_attention_b200_host`` on page-locked host tensors (``"host"``).

Fields of a case: ``E`` batch, ``H`` heads, ``N`` tokens, ``D`` head width, ``B`` block size, ``T``
iterations, ``pad`` side of the zero padding, ``dtype``, ``mask`` (``none``; ``int64`` or ``float``: a quarter
of the sequences right-padded, in the type the language-model callers pass), ``layout`` (``heads``: contiguous
(E, H, N, D) tensors; ``tokens``: (E, H, N, D) views of the (E, N, H, D) projections, result token-major, as the
models call it) and ``scale`` (``rsqrt_d``: N(0, 1/D) as in the op sweep; ``act``: projected hidden states, O(1)
logits with a per-head offset; ``unit``: N(0, 1) with such an offset).
"""
from __future__ import annotations

import math

import torch

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
PEAK_TOKEN_HEADS = 64 * 16 * 1024  # most tokens x heads of one call: the largest batch of the image models
PEAK_WORK = 16 * 65536 * 256       # most tokens x heads x block size: the longest sequence of the op sweep


def _case(name, call, E, H, N, D, B, T, pad, dtype, mask="none", layout="heads", scale="act"):
    return dict(name=name, call=call, E=E, H=H, N=N, D=D, B=B, T=T, pad=pad, dtype=dtype, mask=mask, layout=layout,
                scale=scale)


def listed():
    return [
        # one image through a vision transformer layer: interactive use, latency and launches are all of it
        _case("vit_one_image", "module", 1, 12, 197, 64, 15, 1, "pre", "bf16", layout="tokens"),
        # the op alone in full precision at the smallest benchmark size: a layer while a model is being validated
        _case("op_256_f32", "module", 2, 12, 256, 64, 16, 1, "post", "f32", scale="rsqrt_d"),
        # a vision transformer layer at serving batch (197 tokens: ragged, padded in front)
        _case("vit_batch", "module", 64, 12, 197, 64, 15, 1, "pre", "bf16", layout="tokens"),
        # an encoder layer for text at serving batch; a quarter of the sequences are right-padded
        _case("roberta_batch", "module", 32, 12, 512, 64, 32, 1, "post", "bf16", mask="int64", layout="tokens"),
        # a diffusion transformer layer at 512 x 512, head width 72
        _case("dit_batch", "module", 64, 16, 1024, 72, 32, 2, "pre", "bf16", layout="tokens"),
        # the same model at 256 x 256 sampled in full precision with guidance, the sampler's default iterations
        _case("dit_sample_f32", "module", 8, 16, 256, 72, 16, 3, "pre", "f32", layout="tokens"),
        # long documents padded to the longest of the batch (odd length), summarisation encoder, half precision
        _case("documents_7683_f16", "module", 4, 12, 7683, 64, 64, 2, "post", "f16", mask="float", layout="tokens"),
        # the op sweep over long sequences
        _case("op_4096", "module", 1, 16, 4096, 64, 64, 2, "post", "bf16", scale="rsqrt_d"),
        _case("op_16384", "module", 1, 16, 16384, 64, 128, 2, "post", "bf16", scale="rsqrt_d"),
        _case("op_65536", "module", 1, 16, 65536, 64, 256, 2, "post", "bf16", scale="rsqrt_d"),
        # fine-tuning of the summarisation encoder at 1024 tokens: forward and backward of one layer
        _case("train_1024", "train", 4, 12, 1024, 64, 32, 3, "post", "bf16", mask="float", layout="tokens", scale="unit"),
        # q, k, v and the result in host memory: the copies belong to the call
        _case("host_16384", "host", 1, 16, 16384, 64, 128, 2, "post", "bf16", scale="rsqrt_d"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    call = rng.choice(["module"] * 8 + ["train"] * 2 + ["host"])
    dtype = rng.choice(["bf16"] * 6 + ["f16"] * 2 + ["f32"] * 2)
    D = rng.choice([64] * 5 + [32, 72, 80])
    # sequence lengths: from a short sentence to the longest of the sweep; full precision and training stay with
    # the lengths the models train and validate at, wide heads with those of the image models
    top = {"module": 65536, "train": 4096, "host": 16384}[call]
    if D > 64:
        top = min(top, 4096)
    if dtype == "f32":
        top = min(top, 4096)
    N = _log_int(rng, 64, top)
    if rng.random() < 0.3:             # square sequences, as the sweep and the image models have them
        b = max(8, min(256, round(math.sqrt(N))))
        b = 2 ** round(math.log2(b)) if rng.random() < 0.5 else b
        N = b * b
    else:                              # block size near the square root of the length, ragged end
        b = max(8, min(256, round(math.sqrt(N) * rng.uniform(0.6, 1.4))))
        if rng.random() < 0.5:
            b = 2 ** round(math.log2(b))
        while -(-N // b) > 256:
            b += 1
    H = rng.choice([1, 4, 8, 12, 12, 16, 16])
    room = PEAK_TOKEN_HEADS
    if call == "train" or dtype == "f32":
        room //= 4
    if call == "host":
        room //= 4
    E = _log_int(rng, 1, max(1, min(64, room // (H * N), PEAK_WORK // (H * N * b))))
    T = rng.choice([1, 1, 2, 2, 3])
    if N > 16384:
        T = min(T, 2)                  # as many as the sweep takes at its longest
    masked = rng.random() < 0.4
    return dict(call=call, E=E, H=H, N=N, D=D, B=b, T=T, pad=rng.choice(["pre", "post"]),
                dtype=dtype, mask=rng.choice(["int64", "float"]) if masked else "none",
                layout="heads" if call == "host" else rng.choice(["heads", "tokens"]),
                scale="unit" if call == "train" else rng.choice(["act", "rsqrt_d"]))


def prepare(case, seed):
    from monarch_attention_b200 import MonarchAttention
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    E, H, N, D, dtype = case["E"], case["H"], case["N"], case["D"], DTYPES[case["dtype"]]

    def tensor(std, offset):
        shape = (E, H, N, D) if case["layout"] == "heads" else (E, N, H, D)
        t = torch.randn(shape, generator=g, device=dev)
        t = t if case["layout"] == "heads" else t.permute(0, 2, 1, 3)
        if std != 1.0:
            t *= std
        if offset:
            t += offset * torch.randn(E, H, 1, D, generator=g, device=dev)
        return t.to(dtype)             # strides are kept

    if case["scale"] == "rsqrt_d":
        q, k, v = (tensor(D ** -0.5, 0.0) for _ in range(3))
    else:
        std = 1.5 if case["scale"] == "act" else 1.0
        q, k, v = tensor(std, 0.3), tensor(std, 0.3), tensor(1.0, 0.0)
    mask = None
    if case["mask"] != "none":
        length = torch.full((E, 1), N, device=dev)
        cut = torch.randint(max(1, N // 4), N + 1, (E, 1), generator=g, device=dev)
        length[::4] = cut[::4]
        valid = torch.arange(N, device=dev) < length
        mask = valid.to(torch.int64 if case["mask"] == "int64" else torch.float32)
    state = dict(call=case["call"], q=q, k=k, v=v, mask=mask, T=case["T"], B=case["B"], pre=case["pad"] == "pre")
    if case["call"] == "host":
        for name in ("q", "k", "v"):
            state[name] = torch.empty((E, H, N, D), dtype=dtype, pin_memory=True).copy_(state[name])
        state["out"] = torch.empty((E, H, N, D), dtype=dtype, pin_memory=True)
        state["mask"] = None if mask is None else mask.cpu()
        return state
    module = MonarchAttention(case["B"], case["T"], case["pad"])
    module.token_major_output = case["layout"] == "tokens"
    state["module"] = module
    if case["call"] == "train":
        for name in ("q", "k", "v"):
            state[name].requires_grad_(True)
        state["grad"] = tensor(1.0, 0.0)
    return state


def run(state):
    q, k, v, mask = state["q"], state["k"], state["v"], state["mask"]
    if state["call"] == "host":
        from monarch_attention_b200 import monarch_attention_b200_host
        return monarch_attention_b200_host(q, k, v, mask, state["T"], state["B"], state["pre"], out=state["out"])
    out = state["module"](q, k, v, mask)
    if state["call"] == "train":
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["grad"])
        return {"out": out.detach(), "dq": dq, "dk": dk, "dv": dv}
    return out


def work(case):
    E, H, N, D, B, T = (case[x] for x in ("E", "H", "N", "D", "B", "T"))
    M = -(-N // B)
    size = 4 if case["dtype"] == "f32" else 2
    tensor = E * H * N * D * size
    # contractions of one forward pass: T right-factor, T - 1 left-factor updates, the output product
    flops = E * H * ((T - 1) * 4 * N * D * (B + M) + N * (6 * B * D + 4 * M * D))
    if case["call"] == "train":
        # backward: every contraction has two more; q, k, v, the output's gradient in, three gradients out
        return {"bytes": 4 * tensor + 7 * tensor, "flops": 3 * flops}
    return {"bytes": 4 * tensor, "flops": flops}


def tolerance(case):
    # 16-bit storage between the stages: the roundings of the storage type, carried through up to three iterations
    if case["call"] == "train":
        return {"rel": {"f32": 5e-5, "bf16": 2e-2, "f16": 5e-3}[case["dtype"]]}
    return {"rel": {"f32": 2e-5, "bf16": 1e-2, "f16": 4e-3}[case["dtype"]]}
