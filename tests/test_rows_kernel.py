"""The kernel for TMA shapes at the sizes where its batches, boxes and stores can go wrong, against the oracle: rows
outside the output stay untouched, strides and layouts other than the contiguous one included."""
import pytest
import torch

from oracle import intra_oracle as oracle
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pattern,B,S,H,Hkv,param", [
    ("scatter", 1, 2047, 4, 2, 8), ("scatter", 2, 2049, 3, 3, 8), ("scatter", 1, 1031, 4, 4, 7),   # groups of two lengths
    ("scatter", 1, 300, 2, 1, 299), ("scatter", 1, 128 * 3 + 1, 2, 1, 3),                          # one- and two-token groups; a tile of one row
    ("scatter", 24, 256, 32, 16, 2),          # 768 items of one key tile: a batch of the planner is full on some CTAs
    ("scatter", 80, 200, 32, 32, 8),          # 20480 items: several batches per CTA, the last one partly filled
    ("gather1", 1, 4096, 2, 1, 64), ("gather1", 1, 128 * 128, 2, 2, 128),   # 32-row output boxes inside one segment
    ("gather1", 1, 64 * 9, 4, 2, 8), ("gather1", 3, 16 * 33, 4, 4, 4),
    ("window", 1, 1, 2, 1, 576), ("window", 2, 33, 2, 2, 64), ("window", 1, 4129, 4, 1, 1000), ("window", 1, 575, 3, 1, 65)])
def test_edges(lib, pattern, B, S, H, Hkv, param):
    q, k, v = oracle.make_inputs(B, S, H, Hkv, seed=S + H, device="cuda")
    rc, out = _util.call_fwd(lib, "llm", pattern, q, k, v, param)
    assert rc == 0
    kw = {"window": param} if pattern == "window" else {"group_num": param}
    mask = torch.from_numpy(oracle.build_mask("llm", pattern, S, **kw)).cuda()
    _util.check_against_oracle(out, q, k, v, mask)
    # the same into a (B, H, S + 3, 128) buffer with guard rows between the sequences' rows
    room = torch.full((B, H, S + 3, 128), 7.0, dtype=torch.bfloat16, device="cuda")
    view = room[:, :, 1:S + 1].transpose(1, 2)
    assert _util.call_fwd(lib, "llm", pattern, q, k, v, param, out=view)[0] == 0
    torch.cuda.synchronize()
    assert torch.equal(view, out)
    assert bool((room[:, :, 0] == 7).all()) and bool((room[:, :, S + 1:] == 7).all()), "a row outside the output was written"
    assert _util.device_status(lib) == 0
