"""The work a user of this package has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` builds what a program holds before the call, ``run`` makes one pass through
the public entry points.  The kinds:

* ``train``   ``gate_logits_from_hidden`` + ``nsa_layer`` forward and backward: the layer inside a training step;
* ``module``  ``NSAAttention`` forward and backward with its projections: the drop-in module in a training step;
* ``prefill`` ``nsa_layer`` forward only, block choice returned as well: scoring a prompt;
* ``chunk``   ``module_forward_incremental`` on a chunk of tokens against a key/value cache: chunked prefill;
* ``decode``  ``module_forward_incremental`` token by token against a key/value cache: generation;
* ``window``  ``SlidingWindowAttention`` forward and backward: one branch through its autograd wrapper.

Block sizes, window and slots are the package's defaults (l=32, d=16, l'=64, n=16, w=512) except where the small test
configuration names another window.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "nsa-test_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from nsa import NSAAttention, NSAConfig  # noqa: E402
from nsa.incremental import NSACache, module_forward_incremental  # noqa: E402
from nsa.kernels import SlidingWindowAttention, gate_logits_from_hidden, nsa_layer  # noqa: E402

# head configurations: the paper's (and the benchmark's), one group of 128-wide heads, the small test configuration
HEADS = {"paper": dict(H=64, G=4, dk=192, dv=128, d_model=2560),
         "square": dict(H=32, G=2, dk=128, dv=128, d_model=2048),
         "small": dict(H=8, G=2, dk=64, dv=64, d_model=512)}
L, D, LP, N, W = 32, 16, 64, 16, 512


def listed():
    return [
        # a chat turn being generated: one sequence, 16 tokens one after the other (one of them completes a compressed block)
        dict(name="decode_b1_2k", kind="decode", heads="paper", B=1, cached=2100, steps=16),
        # batched generation over long contexts
        dict(name="decode_b8_32k", kind="decode", heads="paper", B=8, cached=32000, steps=4),
        # a server feeding a long prompt in chunks; the cache does not end on a tile
        dict(name="chunk_512_7k", kind="chunk", heads="paper", B=1, cached=7000, new=512),
        # the repository's first benchmark configuration: fp32 parity-sized training step
        dict(name="train_fp32_512", kind="train", heads="small", dtype="fp32", B=2, T=512, w=256, gate="sigmoid"),
        # the same layer in bf16: the smallest training step, launch-bound
        dict(name="train_bf16_512", kind="train", heads="small", dtype="bf16", B=2, T=512, w=256, gate="sigmoid"),
        # an unpadded batch of short documents: bf16, not a multiple of any tile
        dict(name="train_ragged_1000", kind="train", heads="paper", dtype="bf16", B=1, T=1000, w=W, gate="sigmoid"),
        # a ragged sequence of ordinary length, softmax gates
        dict(name="train_ragged_5001", kind="train", heads="paper", dtype="bf16", B=1, T=5001, w=W, gate="softmax"),
        # the drop-in module in a training step at an ordinary length
        dict(name="module_4k", kind="module", heads="paper", B=1, T=4096),
        # one GPU's share of the batch-sharded training configuration
        dict(name="train_16k", kind="train", heads="paper", dtype="bf16", B=1, T=16384, w=W, gate="sigmoid"),
        # the headline: one 64K sequence, forward and backward
        dict(name="train_64k", kind="train", heads="paper", dtype="bf16", B=1, T=65536, w=W, gate="sigmoid"),
        # the sliding-window configuration: the branch alone
        dict(name="window_b4_8k", kind="window", heads="paper", B=4, T=8192, w=W),
        # the compression/scoring configuration's prompt, forward only
        dict(name="prefill_b2_32k", kind="prefill", heads="paper", B=2, T=32768, w=W),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length, one time in two a multiple of the tile."""
    T = _log(rng, lo, hi)
    return max(128, T // 128 * 128) if rng.random() < 0.5 else T


def draw(rng):
    kind = rng.choice(["decode", "decode", "chunk", "train", "train", "train", "module", "window", "prefill"])
    if kind == "decode":
        B = rng.choice([1, 2, 4, 8])
        return dict(kind=kind, heads="paper", B=B, cached=_log(rng, 64, 262144 // max(B, 4)), steps=rng.randint(1, 16))
    if kind == "chunk":
        return dict(kind=kind, heads=rng.choice(["paper", "square"]), B=rng.choice([1, 1, 2]), cached=_log(rng, 64, 32768),
                    new=_log(rng, 17, 4096))
    if kind == "module":
        return dict(kind=kind, heads=rng.choice(["paper", "square"]), B=rng.choice([1, 2]), T=_length(rng, 2048, 16384))
    if kind == "window":
        B = rng.choice([1, 2, 4])
        return dict(kind=kind, heads=rng.choice(["paper", "square"]), B=B, T=max(256, _log(rng, 256, 32768 // B) // 128 * 128),
                    w=rng.choice([128, 200, 512, 1000]))
    if kind == "prefill":
        B = rng.choice([1, 1, 2])
        return dict(kind=kind, heads=rng.choice(["paper", "square"]), B=B, T=_length(rng, 2048, 65536 // B), w=W)
    if rng.random() < 0.2:
        return dict(kind=kind, heads="small", dtype="fp32", B=rng.choice([1, 2]), T=_log(rng, 64, 1024), w=rng.choice([256, 512]),
                    gate=rng.choice(["sigmoid", "softmax"]))
    heads = rng.choice(["paper", "paper", "square", "small"])
    B = rng.choice([1, 1, 2])
    T = _length(rng, 256, 65536 // B)
    if T % 128 and T < 2048:            # short documents of any length: one at a time, up to 1000 tokens
        B, T = 1, _log(rng, 256, 1000)
    return dict(kind=kind, heads=heads, dtype="bf16", B=B, T=T, w=rng.choice([256, 512]),
                gate=rng.choice(["sigmoid", "sigmoid", "softmax"]))


# ------------------------------------------------------------------------------------------------ inputs

def _config(case):
    h = HEADS[case["heads"]]
    return NSAConfig(d_model=h["d_model"], head_dim_qk=h["dk"], head_dim_v=h["dv"], l=L, d=D, l_prime=LP, n=N,
                     w=case.get("w", W), n_heads=h["H"], n_kv_groups=h["G"], gate_mode=case.get("gate", "sigmoid"))


def _rand(gen):
    def rn(*shape, std=1.0, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype).mul_(std)
    return rn


def _with_block_offsets(rn, x, dim, std=0.5):
    """Adds an offset per 64 positions along ``dim``: blocks differ in importance, as in real sequences."""
    n = x.shape[dim]
    shape = list(x.shape)
    shape[dim] = -(-n // LP)
    off = rn(*shape, std=std, dtype=x.dtype).repeat_interleave(LP, dim=dim)
    return x.add_(off.narrow(dim, 0, n))


def _module(case, rn):
    """NSAAttention in bf16: projections that keep unit variance, compression and gate MLPs N(0, 0.02), zero biases."""
    cfg = _config(case)
    with torch.device("cuda"):
        m = NSAAttention(cfg).bfloat16()
    with torch.no_grad():
        for name, p in m.named_parameters():
            small = name.startswith(("pos_embed", "compress_mlp", "gate_mlp"))
            if p.dim() == 1:
                p.zero_()
            else:
                p.copy_(rn(*p.shape, std=0.02 if small else p.shape[1] ** -0.5))
    return m


def prepare(case, seed):
    h, cfg = HEADS[case["heads"]], _config(case)
    H, G, dk, dv, dm, B = h["H"], h["G"], h["dk"], h["dv"], h["d_model"], case["B"]
    rn = _rand(torch.Generator(device="cuda").manual_seed(seed))
    kind = case["kind"]
    bf = torch.bfloat16
    if kind in ("decode", "chunk"):
        new = case["steps"] if kind == "decode" else case["new"]
        m = _module(case, rn)
        cache = NSACache(cfg, B, case["cached"] + new, "cuda")

        def kv():
            return (_with_block_offsets(rn, rn(B, G, dk, case["cached"], dtype=bf), 3), rn(B, G, case["cached"], dv, dtype=bf))
        k, v = kv()
        cache.append(m._phi_params(), k, v, kv_compress=kv(), kv_sliding=kv())
        return dict(kind=kind, module=m, cache=cache, x=_with_block_offsets(rn, rn(B, new, dm), 1).to(bf))
    if kind == "module":
        m = _module(case, rn)
        x = _with_block_offsets(rn, rn(B, case["T"], dm), 1).to(bf)
        return dict(kind=kind, module=m, x=x.requires_grad_(True), dy=rn(B, case["T"], dm).to(bf))
    dt = torch.float32 if case.get("dtype") == "fp32" else bf
    T = case["T"]
    q = rn(B, H, T, dk).to(dt)
    k = _with_block_offsets(rn, rn(B, G, dk, T), 3).to(dt)
    v = rn(B, G, T, dv).to(dt)
    state = dict(kind=kind, cfg=cfg, q=q, k=k, v=v)
    if kind != "prefill":
        state["do"] = rn(B, H, T, dv).to(dt)
        for t in (q, k, v):
            t.requires_grad_(True)
    if kind != "window":
        state["x"] = rn(B, T, dm).to(dt)
        state["phi"] = (rn(L, L, std=0.02), rn(2 * dk, dk + L, std=0.02), torch.zeros(2 * dk, device="cuda"),
                        rn(dk, 2 * dk, std=0.02), torch.zeros(dk, device="cuda"))
        lin = torch.nn.Linear
        with torch.device("cuda"):
            gate = torch.nn.Sequential(lin(dm, dm // 2), torch.nn.ReLU(), lin(dm // 2, 3 * H)).to(dt)
        with torch.no_grad():
            for p in gate.parameters():
                p.copy_(rn(*p.shape, std=0.02)) if p.dim() > 1 else p.zero_()
        state["gate"] = gate
        if kind == "train":
            for p in state["phi"]:
                p.requires_grad_(True)
    return state


def run(state):
    kind = state["kind"]
    if kind == "decode":
        cache, x = state["cache"], state["x"]
        length, blocks = cache.length, cache.n_blocks
        y = [module_forward_incremental(state["module"], x[:, i:i + 1], cache) for i in range(x.shape[1])]
        cache.length, cache.n_blocks = length, blocks        # the tokens are dropped again, as a rejected draft is
        return y
    if kind == "chunk":
        cache = state["cache"]
        length, blocks = cache.length, cache.n_blocks
        y = module_forward_incremental(state["module"], state["x"], cache)
        cache.length, cache.n_blocks = length, blocks
        return y
    if kind == "module":
        m, x = state["module"], state["x"]
        y, _ = m(x)
        # (the second compression bias shifts all keys alike: its gradient is zero up to rounding and is left out)
        params = [p for name, p in m.named_parameters() if name != "compress_mlp.2.bias"]
        return [y.detach(), *torch.autograd.grad(y, [x, *params], state["dy"])]
    q, k, v, cfg = state["q"], state["k"], state["v"], state["cfg"]
    if kind == "window":
        o = SlidingWindowAttention.apply(q, k, v, q.shape[-1] ** -0.5, cfg.w, cfg)
        return [o.detach(), *torch.autograd.grad(o, [q, k, v], state["do"])]
    if kind == "prefill":
        with torch.no_grad():
            out, info = nsa_layer(q, k, v, gate_logits_from_hidden(state["x"], state["gate"]), state["phi"], cfg, return_info=True)
        return [out, info["indices"]]
    out = nsa_layer(q, k, v, gate_logits_from_hidden(state["x"], state["gate"]), state["phi"], cfg)
    return [out.detach(), *torch.autograd.grad(out, [q, k, v, *state["phi"][:4], *state["gate"].parameters()], state["do"])]


# ------------------------------------------------------------------------------------------------ accounting

def _attention_flops(h, rows, T0, w, backward):
    """Attention FLOPs of query rows at positions T0 + [0, rows) of one sequence, masked keys not counted."""
    t = torch.arange(T0, T0 + rows, dtype=torch.float64)
    keys = {"win": torch.clamp(t + 1, max=w).sum().item(),
            "cmp": torch.clamp(torch.floor((t - L + 1) / D) + 1, min=0).sum().item(),
            "slc": (torch.clamp(torch.floor(t / LP), max=N - 1) * LP + t % LP + 1).sum().item()}
    per_key = 2 * (h["dk"] + h["dv"]) + (2 * (3 * h["dk"] + 2 * h["dv"]) if backward else 0)
    return {b: per_key * h["H"] * c for b, c in keys.items()}


def work(case):
    h, kind, B = HEADS[case["heads"]], case["kind"], case["B"]
    H, G, dk, dv, dm = h["H"], h["G"], h["dk"], h["dv"], h["d_model"]
    es = 4 if case.get("dtype") == "fp32" else 2
    gate_weights = dm * (dm // 2) + (dm // 2) * 3 * H
    proj_weights = dm * (H * dk + 3 * G * (dk + dv)) + H * dv * dm
    if kind == "window":
        T = case["T"]
        tensors = B * T * (2 * H * dk + 2 * H * dv + 2 * G * (dk + dv)) * es
        return dict(bytes=tensors, flops=B * _attention_flops(h, T, 0, case["w"], True)["win"])
    if kind in ("decode", "chunk"):
        new = case["steps"] if kind == "decode" else case["new"]
        passes = new if kind == "decode" else 1
        weights = (proj_weights + gate_weights) * 2
        # per pass: the window's and the selected keys/values, the compressed keys (4-byte) and values once per sequence
        blocks = (case["cached"] + new) // D
        keys = min(case["cached"] + new, W + N * LP if kind == "decode" else 1 << 30)
        cached = B * G * (keys * (dk + dv) * 2 + blocks * (dk * 4 + dv * 2))
        rows = B * new
        f = sum(_attention_flops(h, new, case["cached"], W, False).values()) * B
        return dict(bytes=passes * (weights + cached) + rows * dm * 4, flops=f + 2 * rows * (proj_weights + gate_weights))
    T = case["T"]
    back = kind in ("train", "module")
    flops = B * sum(_attention_flops(h, T, 0, case.get("w", W), back).values())
    flops += 2 * B * T * gate_weights * (3 if back else 1)
    if kind == "module":
        flops += 6 * B * T * proj_weights
        return dict(bytes=B * T * dm * 2 * 4 + 2 * (proj_weights + gate_weights) * 2, flops=flops)
    rows = B * T
    tensors = rows * (H * dk + H * dv + G * (dk + dv)) * es + rows * dm * es + gate_weights * es     # q, out, k, v, x
    if back:
        tensors += rows * (H * dk + H * dv + G * (dk + dv)) * es + gate_weights * es                  # dq, dout, dk, dv
    return dict(bytes=tensors, flops=flops)


def tolerance(case):
    """Four times the errors measured against the same pass in higher precision, relative 2-norm.

    fp32 (against the algorithm in 64 bits on the CPU): 4.5e-6 at the compression weights' gradients, T = 64 to 1000.
    bf16 (against the same inputs through the fp32 kernels): outputs, dQ, dK, dV 2e-3 to 4e-3 and up to 1.1e-2 at the
    compression weights' gradients, which are small sums of large terms; forward-only passes and the window branch 3e-3.
    A row whose n-th and (n+1)-th block scores agree to fp32 rounding may attend the other block (8e-4 of the rows at
    T = 4096), which moves single values of that row by as much as their size.
    """
    if case.get("dtype") == "fp32":
        return dict(rel=2e-5, max=2e-3)
    if case["kind"] == "window":
        return dict(rel=1e-2, max=0.3)
    if case["kind"] in ("train", "module"):
        return dict(rel=3e-2, max=0.99)
    return dict(rel=1.2e-2, max=0.99, differ=1e-2)
