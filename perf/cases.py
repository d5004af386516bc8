"""The workloads this package is measured on: what programs that use it spend their time in.

A language-model server calls the transformers-style attention backend (`llm_backend`) on prompts of any
length and then, token by token, on a growing cache; long-context programs call `intra_llm_attn` on the
three causal patterns; a FLUX-style image transformer alternates the two image patterns through
`flux_joint_attention`. Head counts, group counts, windows and image sizes are those of this repository's
tests and benchmark (32 query heads over 8 KV heads, their eighth for one rank of a head-sharded run, 32
over 32; groups of 2, 3 and 8; windows of 576 and 1000; 64 x 64 and 128 x 128 latents with 24 heads).

`listed()` names the cases, `draw()` gives more of the same ranges, `prepare()` makes the tensors a
program holds before the call, `run()` is one pass, `exact()` the same attention in 64 bits.
"""
import math

import torch

from intra_b200 import intra_llm_attn
from intra_b200.flux import flux_joint_attention
from intra_b200.llm_backend import make_intra_attention

HEAD_DIM = 128
TEXT_LEN = 512


class _Layer:
    """The attention module a model hands to the backend: only its layer index is looked at."""

    def __init__(self, layer_idx):
        self.layer_idx = layer_idx


def _decode(B, S, H=32, Hkv=8, padded=False):
    return {"call": "decode", "B": B, "S": S, "H": H, "Hkv": Hkv, "padded": padded}


def _backend(pattern, B, S, H=32, Hkv=8):
    return {"call": "backend", "pattern": pattern, "B": B, "S": S, "H": H, "Hkv": Hkv}


def _llm(pattern, B, S, param, H=32, Hkv=8, lse=False):
    return {"call": "llm", "pattern": pattern, "B": B, "S": S, "param": param, "H": H, "Hkv": Hkv, "lse": lse}


def _image(pattern, B, width, H=24):
    return {"call": "image", "pattern": pattern, "B": B, "width": width, "H": H}


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # one user's chat in the middle of an answer: a token against a cache of a few thousand, per layer
        named("decode-one", _decode(1, 3001)),
        # a serving batch of answers of different lengths in one padded cache
        named("decode-batch", _decode(16, 8192, padded=True)),
        # a short prompt of arbitrary length on a Scatter layer: latency and launches
        named("prompt-777", _backend("scatter", 1, 777)),
        # the ordinary prompt of the benchmark's smallest configuration
        named("scatter-4k", _llm("scatter", 1, 4096, 8)),
        # a document of arbitrary length: 12345 is no multiple of the 8 groups
        named("scatter-12345", _backend("scatter", 1, 12345)),
        # the Gather-1 pattern at its benchmark length
        named("gather1-16k", _llm("gather1", 1, 16384, 8)),
        # a window layer of the same benchmark configuration
        named("window-16k", _llm("window", 1, 16384, 576)),
        # a long context of odd length whose window part is merged with other keys by its log-sum-exp
        named("window-50001-lse", _llm("window", 1, 50001, 576, lse=True)),
        # the long-context benchmark: a Scatter layer at 65536 tokens
        named("scatter-64k", _llm("scatter", 1, 65536, 8)),
        # image transformer at 1024 x 1024 pixels, both patterns
        named("image-scatter-64", _image("scatter", 1, 64)),
        named("image-gather0-64", _image("gather0", 1, 64)),
        # and at 2048 x 2048 pixels
        named("image-gather0-128", _image("gather0", 1, 128)),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    heads = rng.choice([(32, 8), (32, 8), (32, 32), (4, 1)])
    kind = rng.choice(["decode", "backend", "backend", "llm", "llm", "llm", "image", "image"])
    if kind == "decode":
        B = rng.choice([1, 1, 2, 4, 8, 16, 32])
        S = log_int(64, min(65536, (16 * 8192 * 8) // (B * heads[1])))
        return _decode(B, S, *heads, padded=B > 1 and rng.random() < 0.5)
    if kind == "backend":
        pattern = rng.choice(["scatter", "window"])
        B = rng.choice([1, 1, 2])
        return _backend(pattern, B, log_int(128, 32768 // B), *heads)
    if kind == "llm":
        pattern = rng.choice(["scatter", "gather1", "window"])
        B = rng.choice([1, 1, 2])
        S = log_int(512, 65536 // B)
        if pattern == "gather1":
            S = max(64, S // 64 * 64)
            return _llm(pattern, B, S, 8, *heads, lse=rng.random() < 0.25)
        if pattern == "window":
            return _llm(pattern, B, S, rng.choice([576, 1000]), *heads, lse=rng.random() < 0.25)
        G = rng.choice([2, 3, 8])
        S = min(S, {2: 23000, 3: 28000, 8: 46000}[G] // B)      # ragged groups too: no costlier than the long-context case
        return _llm(pattern, B, S, G, *heads, lse=rng.random() < 0.25)
    # image: whole latents of the two sizes, some or all of the heads (a rank of a sharded run holds a part)
    return _image(rng.choice(["scatter", "gather0"]), rng.choice([1, 2]), rng.choice([64, 64, 128]),
                  rng.choice([3, 6, 8, 12, 24]))


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16)

    call = case["call"]
    state = {"case": case}
    if call == "image":
        # query / key / value of a joint-attention layer, (B, H, S, D), after QK-norm and RoPE
        shape = (case["B"], case["H"], TEXT_LEN + case["width"] ** 2, HEAD_DIM)
        state["qkv"] = [randn(*shape) for _ in range(3)]
        return state
    B, S, H, Hkv = case["B"], case["S"], case["H"], case["Hkv"]
    if call == "llm":
        state["qkv"] = [randn(B, S, H, HEAD_DIM), randn(B, S, Hkv, HEAD_DIM), randn(B, S, Hkv, HEAD_DIM)]
        return state
    # the backend takes (B, H, S, D): here transposed projections of a prompt, or one token and the cache
    state["attention"] = make_intra_attention()
    state["mask"] = None
    if call == "decode":
        state["layer"] = _Layer(0)
        state["qkv"] = [randn(B, H, 1, HEAD_DIM), randn(B, Hkv, S, HEAD_DIM), randn(B, Hkv, S, HEAD_DIM)]
        if case["padded"]:
            # left-padded batch: each sequence fills a share of the cache that ends at the current token
            length = (S * (0.25 + 0.75 * torch.rand(B, generator=g, device="cuda"))).long().clamp_(1, S)
            length[0] = S
            state["mask"] = (torch.arange(S, device="cuda")[None, :] >= (S - length)[:, None])[:, None, None, :]
        return state
    state["layer"] = _Layer(0 if case["pattern"] == "scatter" else 2)
    state["qkv"] = [randn(B, S, n, HEAD_DIM).transpose(1, 2) for n in (H, Hkv, Hkv)]
    return state


def run(state):
    case = state["case"]
    q, k, v = state["qkv"]
    with torch.no_grad():
        if case["call"] == "image":
            return flux_joint_attention(q, k, v, case["pattern"])
        if case["call"] == "llm":
            kw = {"window": case["param"]} if case["pattern"] == "window" else {"group_num": case["param"]}
            return intra_llm_attn(q, k, v, case["pattern"], return_lse=case["lse"], **kw)
        out, _ = state["attention"](state["layer"], q, k, v, state["mask"], scaling=HEAD_DIM ** -0.5)
        return out


def _attended_pairs(case):
    """Query-key pairs of one head of one sequence."""
    if case["call"] == "image":
        W = case["width"]
        n = W * W
        if case["pattern"] == "scatter":
            return (TEXT_LEN + n) * (TEXT_LEN + n // 8)
        return TEXT_LEN * (TEXT_LEN + n // 8) + n * (TEXT_LEN + 256)
    S = case["S"]
    if case["call"] == "decode":
        return S
    pattern = case["pattern"]
    if pattern == "window":
        W = case.get("param", 576)
        full, rest = divmod(S, 64)
        pairs = 0
        for block in range(full + (rest > 0)):
            rows = 64 if block < full else rest
            pairs += rows * min(block * 64, W - 64) + rows * (rows + 1) // 2
        return pairs
    G = case.get("param", 8)
    if pattern == "gather1":
        n = S // G                           # S is a multiple of G * G: every group has S / G tokens
        return G * (n * (n + 1) // 2)
    short, longer = divmod(S, G)
    return longer * ((short + 1) * (short + 2) // 2) + (G - longer) * (short * (short + 1) // 2)


def work(case):
    B, H = case["B"], case["H"]
    Hkv = case.get("Hkv", H)
    if case["call"] == "image":
        S = TEXT_LEN + case["width"] ** 2
    else:
        S = case["S"]
    q_tokens = 1 if case["call"] == "decode" else S
    nbytes = 2 * HEAD_DIM * B * (2 * H * q_tokens + 2 * Hkv * S)
    nbytes += B * S if case.get("padded") else 0
    nbytes += 4 * B * H * S if case.get("lse") else 0
    return {"bytes": nbytes, "flops": 4 * HEAD_DIM * B * H * _attended_pairs(case)}


def tolerance(case):
    # bf16 outputs of fp32 accumulation with probabilities rounded to bf16. Against 64-bit attention on the
    # same inputs, over decode, every causal and image pattern: rel 1.9e-3 .. 2.4e-3, max 6e-3 .. 3.3e-2
    # (log-sum-exp: 4e-7); about four times that.
    return {"rel": 1e-2, "max": 0.12}


def _attend(q, k, v, rows, keys, visible=None, lse=None):
    """64-bit attention of the query tokens `rows` over the key tokens `keys`; tensors are (B, H, S, D)."""
    rep = q.shape[1] // k.shape[1]
    out = torch.empty(q.shape[0], q.shape[1], len(rows), HEAD_DIM, dtype=torch.float64, device=q.device)
    for b in range(q.shape[0]):
        for hk in range(k.shape[1]):
            kk, vv = k[b, hk, keys].double(), v[b, hk, keys].double()
            heads = slice(hk * rep, (hk + 1) * rep)
            s = q[b, heads][:, rows].double() @ kk.T * HEAD_DIM ** -0.5
            if visible is not None:
                s.masked_fill_(~visible, float("-inf"))
            if lse is not None:
                lse[b, heads, rows] = s.logsumexp(-1)
            out[b, heads] = s.softmax(-1) @ vv
    return out


def exact(case, seed):
    state = prepare(case, seed)
    q, k, v = state["qkv"]
    call = case["call"]
    if call == "decode":
        out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
        for b in range(case["B"]):
            keys = torch.arange(case["S"], device="cuda")
            keys = keys if state["mask"] is None else keys[state["mask"][b, 0, 0]]
            one = slice(b, b + 1)
            out[one] = _attend(q[one], k[one], v[one], torch.zeros(1, dtype=torch.long, device="cuda"), keys)
        return out.transpose(1, 2)
    if call == "llm":
        q, k, v = (x.transpose(1, 2) for x in (q, k, v))
    S = q.shape[2]
    pattern = case["pattern"]
    token = torch.arange(S, device="cuda")
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    lse = torch.empty(q.shape[:3], dtype=torch.float64, device="cuda") if case.get("lse") else None

    def attend(rows, keys, visible=None):
        for part in rows.split(2048):                     # bounds the score matrix
            seen = None if visible is None else visible(part[:, None], keys[None, :])
            out[:, :, part] = _attend(q, k, v, part, keys, seen, lse)

    if call == "image":
        W = case["width"]
        text, row, col = token[:TEXT_LEN], (token - TEXT_LEN) // W, (token - TEXT_LEN) % W
        group = torch.where(token < TEXT_LEN, token // 64, row % 2 * 4 + col % 4)
        for g in range(8):
            members = (token >= TEXT_LEN) & (row % 2 * 4 + col % 4 == g)
            rows = group == g if pattern == "scatter" else (token < TEXT_LEN) & (group == g)
            attend(token[rows], torch.cat([text, token[members]]))
        if pattern == "gather0":
            def start(patch):                             # of the 16-wide window around an 8-wide patch
                return min(max(patch * 8 - 4, 0), W - 16)
            for r in range(W // 8):
                for c in range(W // 8):
                    near = (token >= TEXT_LEN) & (row >= start(r)) & (row < start(r) + 16) \
                        & (col >= start(c)) & (col < start(c) + 16)
                    patch = (token >= TEXT_LEN) & (row // 8 == r) & (col // 8 == c)
                    attend(token[patch], torch.cat([text, token[near]]))
        return out
    param = case.get("param", 576 if pattern == "window" else 8)
    if pattern == "window":
        for first in range(0, S, 1024):
            attend(token[first:first + 1024], token[max(0, first - param):first + 1024],
                   lambda i, j: (j <= i) & (j >= i // 64 * 64 - (param - 64)))
    else:
        group = token % param if pattern == "scatter" else token // param % param
        for g in range(param):
            members = token[group == g]
            attend(members, members, lambda i, j: j <= i)
    out = out.transpose(1, 2)
    return out if lse is None else (out, lse)
