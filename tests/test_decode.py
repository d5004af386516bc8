"""One-token decode of the transformers-style backend: the decode kernel against fp64 attention and against
the SDPA call it stands in for, over the forms of cache and mask it takes; what it leaves to SDPA."""
import ctypes

import numpy as np
import pytest
import torch
import torch.nn.functional as F
from torch.overrides import TorchFunctionMode

from intra_b200 import interface, intra_llm_attn
from intra_b200.interface import decode_attn
from intra_b200.llm_backend import make_intra_attention


def _inputs(B, H, Hkv, S, seed=0, layout="bhsd", device="cuda"):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, H, 1, 128, generator=g).to(torch.bfloat16).to(device)
    shape = {"bhsd": (B, Hkv, S, 128), "bshd": (B, S, Hkv, 128), "sliced": (B, Hkv, S + 40, 128), "batch1": (1, Hkv, S, 128)}[layout]
    k, v = (torch.randn(*shape, generator=g).to(torch.bfloat16).to(device) for _ in range(2))
    if layout == "bshd":
        k, v = k.transpose(1, 2), v.transpose(1, 2)
    if layout == "sliced":                                   # a cache that is longer than what is filled
        k[:, :, :3], v[:, :, :3], k[:, :, S + 3:], v[:, :, S + 3:] = (float("nan"),) * 4
        k, v = k[:, :, 3:S + 3], v[:, :, 3:S + 3]
    if layout == "batch1":
        k, v = k.expand(B, -1, -1, -1), v.expand(B, -1, -1, -1)
    return q, k, v


def _mask(kind, B, S, device="cuda"):
    g = torch.Generator().manual_seed(7)
    if kind is None:
        return None
    if kind == "left-padded":
        start = (S * 0.75 * torch.rand(B, 1, generator=g)).long()
        start[0] = 0
        m = torch.arange(S)[None, :] >= start
    elif kind == "one-key":
        m = torch.arange(S)[None, :].expand(B, S) == torch.randint(S, (B, 1), generator=g)
    else:
        m = torch.rand(1 if kind == "shared" else B, S, generator=g) < 0.3
        m[:, -1] = True
    if kind == "strided":
        wide = torch.zeros(m.shape[0], 2 * S + 5, dtype=torch.bool)
        wide[:, 5::2] = m
        return wide.to(device)[:, None, None, 5::2]
    if kind == "longer":                                     # cut to the cache's length by the backend's contract
        m = torch.cat([m, torch.ones(m.shape[0], 9, dtype=torch.bool)], 1)
    return m.to(device)[:, None, None, :]


def _reference(q, k, v, mask, scale):
    """fp64 result and sum_j p_j |v_j|, both (B, 1, H, 128)."""
    rep = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(rep, 1).double(), v.repeat_interleave(rep, 1).double()
    s = (q.double() @ k.transpose(-1, -2)) * scale
    if mask is not None:
        s = s.masked_fill(~mask[..., : k.shape[2]], float("-inf"))
    p = s.softmax(-1)
    return (p @ v).transpose(1, 2), (p @ v.abs()).transpose(1, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,Hkv,S,layout,mask", [
    (1, 32, 8, 1, "bhsd", None), (1, 32, 8, 15, "bhsd", None), (1, 32, 8, 17, "bshd", None),       # ends of a 16-key block
    (1, 4, 1, 63, "bhsd", "random"), (2, 32, 8, 64, "sliced", None), (3, 32, 8, 65, "batch1", "shared"),
    (1, 32, 8, 1008, "bhsd", None), (1, 32, 8, 1009, "bhsd", None), (1, 32, 8, 3001, "bshd", None),   # clusters of 8, of 16
    (1, 32, 8, 8176, "bhsd", None), (5, 32, 8, 300, "bhsd", "random"),                               # the last of 16; of 4
    (16, 16, 8, 8192, "batch1", "left-padded"),               # 2 CTAs a unit would do, 4 are needed: 128 blocks each, all they can list
    (8, 8, 8, 16384, "batch1", "random"), (8, 16, 8, 16400, "batch1", "random"),    # 8 are full; one block more takes a second cluster
    (1, 32, 8, 8191, "bhsd", None), (1, 4, 1, 40000, "sliced", None),                                 # several clusters
    (16, 32, 8, 2100, "bhsd", "left-padded"), (20, 32, 32, 300, "bhsd", "random"), (3, 32, 32, 70, "bhsd", None), (300, 4, 1, 40, "bhsd", "one-key"),
    (2, 9, 1, 500, "bhsd", "random"), (2, 36, 2, 77, "bhsd", "strided"), (1, 64, 2, 5000, "bshd", "longer"),   # 9, 18, 32 heads per KV head
    (40, 16, 8, 2500, "bhsd", "random")])
def test_decode_kernel_vs_fp64(B, H, Hkv, S, layout, mask):
    q, k, v = _inputs(B, H, Hkv, S, layout=layout)
    m = _mask(mask, B, S)
    out = decode_attn(q, k, v, m, 0.1)
    assert out is not None and out.shape == (B, 1, H, 128) and out.is_contiguous()
    ref, spread = _reference(q, k, v, m, 0.1)
    # half a bf16 ulp of the result (2^-8 |ref| covers it twice) + probabilities kept to 16 bits and fp32 sums:
    # 2^-16 each, a factor four of margin
    excess = (out.double() - ref).abs() - (2.0 ** -8 * ref.abs() + 2.0 ** -14 * spread)
    assert float(excess.max()) <= 0
    assert torch.equal(out, decode_attn(q, k, v, m, 0.1)), "two runs differ"
    fn = make_intra_attention()
    got, w = fn(None, q, k, v, m, scaling=0.1)
    assert w is None and torch.equal(got, out)
    rep = H // Hkv
    sdpa = F.scaled_dot_product_attention(q, k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1),
                                          attn_mask=None if m is None else m[..., :S], scale=0.1).transpose(1, 2)
    worst = (out.double() - sdpa.double()).abs() - (2.0 ** -7 * ref.abs() + 2.0 ** -7 * spread)   # SDPA rounds P to bf16
    assert float(worst.max()) <= 0


@pytest.mark.gpu
def test_decode_kernel_masked_keys_and_special_values():
    q, k, v = _inputs(2, 8, 2, 200)
    m = _mask("random", 2, 200)
    clean = decode_attn(q, k, v, m)
    k2, v2 = k.clone(), v.clone()
    hidden = ~m[:, 0, 0, :]
    k2[hidden[:, None].expand(2, 2, 200)] = float("nan")
    v2[hidden[:, None].expand(2, 2, 200)] = float("inf")
    assert torch.equal(decode_attn(q, k2, v2, m), clean), "a hidden key's row reached the result"
    m0 = m.clone()
    m0[1] = False                                              # a sequence that sees nothing
    out = decode_attn(q, k, v, m0)
    assert torch.equal(out[0], clean[0]) and not bool(out[1].any())
    k3 = k.clone()
    k3[0, :, 50] = float("nan")                                # a visible NaN reaches every head of its batch entry only
    out = decode_attn(q, k3, v)
    assert bool(out[0].isnan().all()) and bool(torch.isfinite(out[1]).all())
    v3 = v.clone()                                             # visible infinities stay infinities, in their dimension only
    v3[0, 0, 50, 5], v3[0, 1, 7, 9], v3[1, 0, 0, 127] = float("inf"), float("-inf"), float("-inf")
    out = decode_attn(q, k, v3)
    ref, spread = _reference(q, k, v3, None, 128 ** -0.5)
    finite = ref.isfinite()
    assert int((~finite).sum()) == 3 * 4 and torch.equal(out.double()[~finite], ref[~finite])
    assert float(((out.double() - ref).abs() - (2.0 ** -8 * ref.abs() + 2.0 ** -14 * spread))[finite].max()) <= 0
    v3[0, 0, 60, 5] = float("-inf")                            # both signs: undefined
    assert bool(decode_attn(q, k, v3)[0, 0, :4, 5].isnan().all())
    one = decode_attn(q[:1], k[:1, :, :1], v3[1:, :, :1])      # a single key: its probability is exactly one
    assert torch.equal(one[0, 0], v3[1, :, 0].repeat_interleave(4, 0))
    big = decode_attn(q * 50, k, v)                            # near one-hot rows
    ref, spread = _reference(q * 50, k, v, None, 128 ** -0.5)
    assert float(((big.double() - ref).abs() - (2.0 ** -8 * ref.abs() + 2.0 ** -11 * spread)).max()) <= 0   # fp32 scores of several hundred


@pytest.mark.gpu
def test_decode_kernel_under_capture_and_on_other_streams():
    cases = [_inputs(1, 32, 8, 3001, seed=1), _inputs(1, 4, 1, 40000, seed=2)]
    want = [decode_attn(*c) for c in cases]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = [decode_attn(*c) for c in cases]
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [decode_attn(*c) for c in cases]
    for x in got:
        x.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,S,masked,kernel", [
    (1, 8, 900, False, True), (1, 8, 6900, False, False), (1, 24, 3500, False, True), (2, 32, 1350, False, False),
    (1, 32, 6100, False, True), (1, 32, 6110, False, False), (16, 32, 100, False, True), (16, 32, 110, False, False),
    (20, 32, 300, False, False), (32, 32, 20, False, False), (128, 32, 32, True, False), (128, 32, 33, True, True),
    (64, 32, 32, True, True)])
def test_multi_head_caches_go_where_they_are_quicker(B, H, S, masked, kernel):
    q, k, v = _inputs(B, H, H, S)
    m = _mask("left-padded", B, S) if masked else None
    fn = make_intra_attention()
    want = decode_attn(q, k, v, m) if kernel else F.scaled_dot_product_attention(q, k, v, attn_mask=m).transpose(1, 2)
    out = fn(None, q, k, v, m)[0]
    assert torch.equal(out, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = fn(None, q, k, v, m)[0]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(replayed, out)


@pytest.mark.gpu
def test_a_failed_launch_is_reported_once(lib):
    """A decode launch that the runtime refuses (on a stream whose capture has been invalidated) returns its error; the
    next attention call on the thread succeeds."""
    q, k, v = _inputs(1, 32, 8, 100)
    want, out = decode_attn(q, k, v), torch.empty(1, 1, 32, 128, dtype=torch.bfloat16, device="cuda")
    prompt = torch.randn(1, 64, 4, 128, device="cuda").bfloat16()
    with torch.no_grad():                            # a first attention call sets the device up, which forgets errors
        prefill = intra_llm_attn(prompt, prompt, prompt, "window")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so.%s" % torch.version.cuda.split(".")[0])        # the runtime torch has loaded
    raw, graph, need = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_int64(0)

    def decode(s):
        return lib.intra_b200_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), None, out.data_ptr(), None, 0, need, 1, 100, 32, 8,
                                     *q.stride()[:2], k.stride(0), k.stride(2), k.stride(1), v.stride(0), v.stride(2), v.stride(1),
                                     0, 0, 128 ** -0.5, 0, s)

    assert rt.cudaStreamBeginCapture(raw, 2) == 0                                   # 2: this thread may call anything meanwhile
    assert rt.cudaStreamSynchronize(raw) != 0                                       # not allowed: the capture is invalid now
    rc = decode(raw)
    assert rt.cudaStreamEndCapture(raw, ctypes.byref(graph)) != 0
    rt.cudaGetLastError()
    assert rc == -4 and lib.intra_b200_last_cuda_error() != 0
    with torch.no_grad():
        assert torch.equal(intra_llm_attn(prompt, prompt, prompt, "window"), prefill)
    assert decode(None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.gpu
def test_calls_the_decode_kernel_leaves_to_sdpa():
    q, k, v = _inputs(2, 8, 2, 64)
    m = _mask("random", 2, 64)
    fn = make_intra_attention()

    def same_as_sdpa(q, k, v, m=None):
        assert decode_attn(q, k, v, m) is None
        rep = q.shape[1] // k.shape[1]
        want = F.scaled_dot_product_attention(q, k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1), attn_mask=m).transpose(1, 2)
        assert torch.equal(fn(None, q, k, v, m)[0], want)

    same_as_sdpa(q.half(), k.half(), v.half())
    same_as_sdpa(q[..., :64], k[..., :64], v[..., :64])
    same_as_sdpa(q, k, v, torch.zeros(2, 1, 1, 64, device="cuda", dtype=torch.bfloat16))
    same_as_sdpa(q, k, v, m.expand(2, 8, 1, 64))                               # a mask per head
    same_as_sdpa(q, k.clone().requires_grad_(True), v)
    wide = torch.randn(2, 2, 64, 132, device="cuda").bfloat16()[..., 2:130]     # rows that are not 16-byte aligned
    same_as_sdpa(q, wide, v)
    assert decode_attn(q, k, v, None, torch.tensor(0.1)) is None                # a scale that is a tensor: SDPA's to take or to refuse
    with pytest.raises(TypeError):
        fn(None, q, k, v, scaling=torch.tensor([0.1]))
    assert torch.equal(decode_attn(q, k, v, None, np.float32(0.125)), decode_attn(q, k, v, None, 0.125))
    with torch.autocast("cuda", dtype=torch.float16):
        assert decode_attn(q, k, v) is None and fn(None, q, k, v)[0].dtype == torch.float16
    batched = torch.vmap(lambda a, b, c: fn(None, a, b, c)[0])(q[None], k[None], v[None])
    assert float((batched[0].float() - decode_attn(q, k, v).float()).abs().max()) <= 1.6e-2


@pytest.mark.gpu
def test_decode_on_another_gpu_is_sdpa(monkeypatch):
    """The library refuses devices that are not sm_100; the step runs there as torch operators."""
    class Refuses:
        intra_b200_decode = staticmethod(lambda *args: -5)

    q, k, v = _inputs(2, 8, 2, 64)
    monkeypatch.setattr(interface, "lib", Refuses)
    want = F.scaled_dot_product_attention(q, k.repeat_interleave(4, 1), v.repeat_interleave(4, 1)).transpose(1, 2)
    assert decode_attn(q, k, v) is None
    assert torch.equal(make_intra_attention()(None, q, k, v)[0], want)


@pytest.mark.parametrize("name", ["_tracing_state", "_dispatch_modes", "_functorch_level", "_forward_ad", "_function_modes"])
def test_a_torch_without_a_private_name_is_taken_to_be_watching(monkeypatch, name):
    assert not interface._watched()
    monkeypatch.setattr(interface, name, None)
    assert interface._watched()


class _Calls(TorchFunctionMode):
    """Notes the functions that are called under it."""

    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


def test_function_modes_watch_and_default_devices_do_not():
    with torch.device("cpu"):
        assert not interface._watched()
        with _Calls():
            assert interface._watched()
    with _Calls(), torch.device("cpu"):
        assert interface._watched()


@pytest.mark.gpu
def test_a_function_mode_sees_the_decode_step():
    q, k, v = _inputs(2, 8, 2, 64)
    want = decode_attn(q, k, v)
    with torch.device("cuda"):
        assert torch.equal(decode_attn(q, k, v), want)
    with _Calls() as calls:
        make_intra_attention()(None, q, k, v)
    assert F.scaled_dot_product_attention in calls.seen


def test_names_torch_does_not_have():
    assert interface._torch_name("_C._no_such_name") is None and interface._torch_name("no_module.no_name") is None
    assert interface._torch_name("nn.functional.scaled_dot_product_attention") is F.scaled_dot_product_attention


@pytest.mark.gpu
def test_decode_without_torchs_private_names(monkeypatch):
    q, k, v = _inputs(2, 8, 2, 64)
    want = decode_attn(q, k, v)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert interface._raw_stream(0) == side.cuda_stream
    monkeypatch.setattr(interface, "_raw_stream", lambda index: torch.cuda.current_stream(index).cuda_stream)
    assert torch.equal(decode_attn(q, k, v), want)
    monkeypatch.setattr(interface, "_functorch_level", None)
    sdpa = F.scaled_dot_product_attention(q, k.repeat_interleave(4, 1), v.repeat_interleave(4, 1)).transpose(1, 2)
    assert torch.equal(make_intra_attention()(None, q, k, v)[0], sdpa)


def test_decode_on_the_cpu_is_sdpa():
    q, k, v = _inputs(2, 8, 2, 30, device="cpu")
    m = _mask("random", 2, 30, device="cpu")
    assert decode_attn(q, k, v, m) is None
    out, _ = make_intra_attention()(None, q, k, v, m)
    want = F.scaled_dot_product_attention(q, k.repeat_interleave(4, 1), v.repeat_interleave(4, 1), attn_mask=m).transpose(1, 2)
    assert torch.equal(out, want)
