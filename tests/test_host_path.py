"""The native host path (``_host``) against the descriptor wrappers it stands in for: the same kernels with the same
arguments, so every output is bit-identical."""

import pytest
import torch

from tests.helpers import zoo_inputs
from tests.test_ssd_ops import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,K,V,dtype", [("simple_gla", 128, 64, torch.float16), ("gla", 64, 64, torch.bfloat16),
                                            ("delta", 128, 128, torch.bfloat16), ("kda", 64, 128, torch.float16)])
@pytest.mark.parametrize("form", ["plain", "converted"])
def test_zoo_cells(cell, K, V, dtype, form):
    from linquant_b200.kernels import zoo

    fn = getattr(zoo, f"chunk_{cell}_int8")
    delta, diag = cell in ("delta", "kda"), cell in ("gla", "kda")
    B, T, H = 2, 192, 3
    q, k, v, g, beta = (None if t is None else t.cuda() for t in zoo_inputs(
        B, T, H, K, V, decay="diagonal" if diag else "scalar", delta=delta, dtype=dtype, seed=4))
    full = lambda *s: torch.rand(*s, device="cuda") * 0.01 + 0.005  # noqa: E731
    sc = {"q": full(H), "k": full(H), "kw": full(H, K), "vw": full(H, V), "vl": full(H, V), "state": full(H, V),
          "w": full(H), "el": full(H, V), "ew": full(H, V)}
    kw = dict(rot=torch.ones(K, device="cuda"), output_final_state=True, initial_state=torch.randn(B, H, K, V, device="cuda") * 0.1)
    if form == "converted":  # strided activations, half-precision gates and expanded scales: a dense copy is made of each
        q, v = q.transpose(1, 2).contiguous().transpose(1, 2), v.transpose(1, 2).contiguous().transpose(1, 2)
        g = g.half()
        sc = {n: t[:, :1].expand(t.shape) if t.dim() == 2 else t.double() for n, t in sc.items()}
        kw["rot"] = kw["rot"].cpu()
    args = (q, k, v, g) + ((beta,) if delta else ())
    o, s = fn(*args, sc, **kw)
    o2, s2 = fn(*args, sc, **kw, _debug={})
    assert torch.equal(o, o2) and torch.equal(s, s2) and o.dtype == dtype and float(o.float().abs().max()) > 0


@pytest.mark.parametrize("cell", ["gla", "kda"])
@pytest.mark.parametrize("offset", [1, 2])
def test_per_channel_decay_at_an_odd_address(cell, offset):
    """A dense slice of a flat gate buffer that starts off a 16-byte boundary gives what an aligned copy of it gives."""
    from linquant_b200.kernels import zoo

    B, T, H, K, V = 1, 128, 2, 64, 64
    q, k, v, g, beta = (t.cuda() for t in zoo_inputs(B, T, H, K, V, decay="diagonal", delta=True, dtype=torch.bfloat16, seed=6))
    flat = torch.empty(g.numel() + 4, device="cuda")
    odd = flat[offset:offset + g.numel()].view(g.shape).copy_(g)
    assert odd.is_contiguous() and odd.data_ptr() % 16
    full = lambda *s: torch.full(s, 0.01, device="cuda")  # noqa: E731
    sc = {"q": full(H), "k": full(H), "kw": full(H, K), "vw": full(H, V), "vl": full(H, V), "state": full(H, V),
          "w": full(H), "el": full(H, V), "ew": full(H, V)}
    extra = (beta,) if cell == "kda" else ()
    fn = getattr(zoo, f"chunk_{cell}_int8")
    want, _ = fn(q, k, v, g, *extra, sc)
    for debug in (None, {}):
        got, _ = fn(q, k, v, odd, *extra, sc, _debug=debug)
        assert torch.equal(got, want)


@pytest.mark.parametrize("cell", ["simple_gla", "gla", "delta", "kda"])
def test_a_refused_launch_is_reported_once(cell):
    """More (batch, head) pairs than a grid has rows: the launch is refused on the host. The next call, and torch's own next launch,
    must not find that error."""
    from linquant_b200 import _cabi
    from linquant_b200.kernels import zoo

    delta, diag, K = cell in ("delta", "kda"), cell in ("gla", "kda"), 64

    def call(B, H):
        zero = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device="cuda")  # noqa: E731
        q, k, v = (zero(B, 64, H, K, dtype=torch.bfloat16) for _ in range(3))
        sc = {n: zero(H) + 1 for n in ("q", "k", "w")} | {n: zero(H, K) + 1 for n in ("kw", "vl", "vw", "state", "el", "ew")}
        g = zero(B, 64, H, K) if diag else zero(B, 64, H)
        return getattr(zoo, f"chunk_{cell}_int8")(q, k, v, g, *((zero(B, 64, H),) if delta else ()), sc)[0]

    with pytest.raises(_cabi.LinQuantError, match="invalid configuration"):
        call(4100, 16)
    assert float((call(1, 2) + 1).abs().max()) == 1.0


def test_zoo_errors():
    from linquant_b200 import _cabi
    from linquant_b200.kernels.zoo import chunk_simple_gla_int8

    q, k, v, g, _ = (None if t is None else t.cuda() for t in zoo_inputs(1, 96, 2, 64, 64, decay="scalar"))
    one = {"q": torch.ones(2).cuda(), "k": torch.ones(2).cuda(), "kw": torch.ones(2, 64).cuda(), "state": torch.ones(2, 64).cuda()}
    with pytest.raises(AssertionError):
        chunk_simple_gla_int8(q, k, v, g, one)
    with pytest.raises(_cabi.LinQuantError):  # no value scales
        chunk_simple_gla_int8(q[:, :64], k[:, :64], v[:, :64], g[:, :64], one)
    with pytest.raises(NotImplementedError):
        chunk_simple_gla_int8(q[:, :64].double(), k[:, :64].double(), v[:, :64].double(), g[:, :64], one)


@pytest.mark.parametrize("chunk,N,G,L", [(256, 128, 1, 256), (128, 128, 2, 384), (192, 64, 2, 576), (64, 64, 1, 320)])
@pytest.mark.parametrize("keyside", [False, True])
def test_ssd_combined(chunk, N, G, L, keyside, monkeypatch):
    from linquant_b200.kernels.mamba2 import ssd_combined as sc

    k = {n: t.cuda() if torch.is_tensor(t) else t for n, t in make_case(B=2, L=L, H=6, G=G, N=N, chunk=chunk, seed=5).items()}
    one = torch.ones(1, device="cuda")

    def call(D, D_scale, dt_scale):
        return sc._quant_mamba_chunk_scan_combined_fwd(
            k["x"], k["dt_raw"], dt_scale, k["A_log"], dt_scale, k["qB"], k["sB"], k["qC"], k["sC"], chunk, D, D_scale,
            static_state_scale=k["state_scale"], static_cb_scale=k["cb_scale"], alpha_hp=k["alpha"],
            bscale_g=k["sB"], keyside=keyside, x_scale_hp=k["x_scale"], b_fp=k["Bm"], b_gate_scale=k["b_gate"])[0]

    forms = [(k["D"], 1.0, 1.0), (k["D"].half(), 0.5, one), (k["D"].unsqueeze(1).expand(6, 64), one * 0.5, one), (None, 1.0, 1.0)]
    native = [call(*f) for f in forms]
    monkeypatch.setattr(sc, "_SUB_OPS", ())  # what a caller that replaces a sub-op gets: the wrappers one by one
    for f, got in zip(forms, native):
        want = call(*f)
        assert got.dtype == torch.float16 and torch.equal(got, want) and float(want.float().abs().max()) > 0
