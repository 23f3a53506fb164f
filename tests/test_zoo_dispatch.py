"""Tile choices that follow the number of (batch, head) pairs: a batch large enough for the throughput variants gives, bit for
bit, what its elements give one at a time through the small-problem variants (which the oracle tests cover)."""

import pytest
import torch

from tests.helpers import zoo_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,B,H,K,V,NT", [
    ("simple_gla", 5, 10, 128, 64, 5),   # 200 CTAs of 64 key channels: three chunks in flight
    ("simple_gla", 10, 8, 64, 128, 3),   # 320: one in flight
    ("gla", 3, 20, 64, 128, 2),          # 240
    ("gla", 5, 16, 128, 64, 1),          # 320
    ("delta", 5, 8, 128, 128, 3),        # 320 groups of 16 value rows: two per CTA
    ("delta", 10, 8, 64, 64, 1),
    ("kda", 5, 8, 128, 128, 4),
    ("kda", 10, 8, 64, 64, 2),
])
def test_large_batch_equals_its_elements(cell, B, H, K, V, NT):
    from linquant_b200.kernels import zoo

    fn = getattr(zoo, f"chunk_{cell}_int8")
    delta, diag = cell in ("delta", "kda"), cell in ("gla", "kda")
    q, k, v, g, beta = (None if t is None else t.cuda() for t in zoo_inputs(
        B, 64 * NT, H, K, V, decay="diagonal" if diag else "scalar", delta=delta, dtype=torch.bfloat16, seed=8))
    full = lambda *s: torch.rand(*s, device="cuda") * 0.01 + 0.005  # noqa: E731
    sc = {"q": full(H), "k": full(H), "kw": full(H, K), "vw": full(H, V), "vl": full(H, V), "state": full(H, V),
          "w": full(H), "el": full(H, V), "ew": full(H, V)}
    s0 = torch.randn(B, H, K, V, device="cuda") * 0.1
    args = (q, k, v, g) + ((beta,) if delta else ())
    kw = dict(rot=torch.ones(K, device="cuda"), output_final_state=True)
    o, s = fn(*args, sc, initial_state=s0, **kw)
    assert float(o.float().abs().max()) > 0
    for b in range(B):
        ob, sb = fn(*(t[b:b + 1] for t in args), sc, initial_state=s0[b:b + 1], **kw)
        assert torch.equal(o[b:b + 1], ob) and torch.equal(s[b:b + 1], sb), f"element {b}"
