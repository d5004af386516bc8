"""The Python call path: both axis orders, layouts that are read in place and layouts that are copied, no memory of
tensors between calls."""
import pytest
import torch

from intra_b200 import intra_image_attn, intra_llm_attn
from intra_b200.flux import flux_joint_attention
from intra_b200.llm_backend import make_intra_attention

pytestmark = pytest.mark.gpu


class _Layer:
    def __init__(self, layer_idx):
        self.layer_idx = layer_idx


def _layouts(x):
    """(B, S, H, 128) views of x's values in the layouts a caller may hold; the last two have to be copied."""
    yield "contiguous", x.contiguous()
    yield "heads-first", x.transpose(1, 2).contiguous().transpose(1, 2)
    wide = torch.zeros(x.shape[0], x.shape[1] + 5, x.shape[2] + 1, 136, dtype=x.dtype, device=x.device)
    wide[:, 2:-3, 1:, :128] = x
    yield "sliced", wide[:, 2:-3, 1:, :128]
    odd = torch.zeros(x.shape[0], x.shape[1], x.shape[2], 132, dtype=x.dtype, device=x.device)
    odd[..., 2:130] = x
    yield "misaligned", odd[..., 2:130]
    yield "strided", x.transpose(1, 3).contiguous().transpose(1, 3)


@pytest.mark.parametrize("S", [200, 643])
def test_layouts_and_axis_orders(S):
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(2, S, n, 128, generator=g, device="cuda").bfloat16() for n in (4, 2, 2))
    backend = make_intra_attention()
    with torch.no_grad():
        want = {p: intra_llm_attn(q, k, v, p) for p in ("scatter", "window")}
        for (name, ql), (_, kl), (_, vl) in zip(_layouts(q), _layouts(k), _layouts(v)):
            for layer, pattern in ((0, "scatter"), (2, "window")):
                out, lse = intra_llm_attn(ql, kl, vl, pattern, return_lse=True)
                assert out.shape == q.shape and torch.equal(out, want[pattern]), (name, pattern)
                got, w = backend(_Layer(layer), *(x.transpose(1, 2) for x in (ql, kl, vl)))
                assert w is None and got.shape == q.shape and torch.equal(got, want[pattern]), (name, pattern)
    # the backend takes tensors that require gradients (its result does not); the entry point refuses them
    qr = q.transpose(1, 2).detach().requires_grad_(True)
    out, _ = backend(_Layer(0), qr, k.transpose(1, 2), v.transpose(1, 2))
    assert not out.requires_grad and torch.equal(out, want["scatter"])
    with pytest.raises(RuntimeError, match="forward-only"):
        intra_llm_attn(q.detach().requires_grad_(True), k, v)


def test_image_axis_orders():
    q, k, v = (torch.randn(1, 512 + 64 * 64, 3, 128, device="cuda").bfloat16() for _ in range(3))
    with torch.no_grad():
        for pattern in ("scatter", "gather0"):
            want = intra_image_attn(q, k, v, pattern, 64)
            for (_, ql), (_, kl), (_, vl) in zip(_layouts(q), _layouts(k), _layouts(v)):
                out = flux_joint_attention(ql.transpose(1, 2), kl.transpose(1, 2), vl.transpose(1, 2), pattern)
                assert out.shape == (1, 3, 512 + 64 * 64, 128) and torch.equal(out.transpose(1, 2), want)


def test_same_addresses_other_shapes_and_values():
    room = torch.randn(1, 640, 4, 128, device="cuda").bfloat16()
    with torch.no_grad():
        a = intra_llm_attn(room, room, room, "window")
        b = intra_llm_attn(room[:, :64], room[:, :64], room[:, :64], "window")
        assert torch.equal(a[:, :64], b)
        room.mul_(0.5)
        assert torch.equal(intra_llm_attn(room, room, room, "window"), intra_llm_attn(room.clone(), room.clone(), room.clone(), "window"))
