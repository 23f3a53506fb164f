"""The WY prologues where their operand paths differ: keys in fp32 (D_QK without a rotation), keys as two bf16 pieces (fp16),
fp32 rows rotated as three pieces, and decays so strong that a diagonal block cannot be factored around its first row."""

import pytest
import torch

from tests import test_zoo_delta as delta
from tests import test_zoo_diag as diag
from tests.helpers import OracleRun, code_mismatch, rel_l2, zoo_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,K,V,dqk,sigma", [
    (torch.float16, 128, 128, True, 0.5),
    (torch.bfloat16, 64, 128, True, 1.0),
    (torch.float16, 64, 64, False, 0.5),
    (torch.bfloat16, 128, 128, False, 1.0),
])
def test_delta_rotated_operands(dtype, K, V, dqk, sigma):
    q, k, v, g, beta = zoo_inputs(1, 192, 3, K, V, decay="scalar", delta=True, dtype=dtype, seed=3)
    d = torch.logspace(-0.5, 0.5, K).expand(3, K).contiguous() if dqk else None
    delta.run_case(q, k, v, g, beta, policy="kernel_ptk", sigma=sigma, rot=True, dqk=d, label=f"{dtype} K={K} V={V} dqk={dqk}")


@pytest.mark.parametrize("dtype,K,V", [(torch.bfloat16, 128, 128), (torch.float16, 64, 128), (torch.float16, 128, 64), (torch.bfloat16, 64, 64)])
def test_delta_unrounded_keys(dtype, K, V):
    """D_QK without a rotation keeps q D and k / D in fp32. With powers of two they are exact in the activation dtype, and the
    call equals one on inputs scaled beforehand: same codes of q and k, W and the output up to rounding boundaries."""
    from linquant_b200.kernels.zoo import chunk_delta_int8

    q, k, v, g, beta = (t.cuda() for t in zoo_inputs(1, 192, 3, K, V, decay="scalar", delta=True, dtype=dtype, seed=5))
    d = torch.tensor([0.5, 1.0, 2.0, 1.0], device="cuda").repeat(3, K // 4)
    qs, ks = (q.float() * d).to(dtype), (k.float() / d).to(dtype)
    sc = OracleRun(qs.cpu(), ks.cpu(), v.cpu(), g.cpu(), beta.cpu(), family="delta", decay="scalar", sigma=0.5).scales("cuda")
    got, want = {}, {}
    o, s = chunk_delta_int8(q, k, v, g, beta, sc, sigma=0.5, output_final_state=True, dqk=d, _debug=got)
    o2, s2 = chunk_delta_int8(qs, ks, v, g, beta, sc, sigma=0.5, output_final_state=True, _debug=want)
    for name in ("qq", "kl", "kwT"):
        assert torch.equal(got["workspace"].view(name), want["workspace"].view(name)), name
    code_mismatch(got["workspace"].view("wq"), want["workspace"].view("wq"), "W codes")
    # one flipped code of W moves an output by less than its own rounding: the bound the oracle comparisons use
    assert rel_l2(o, o2) <= 2e-3 and rel_l2(s, s2) <= 1e-3


@pytest.mark.parametrize("dtype,K,V", [(torch.bfloat16, 128, 128), (torch.float16, 64, 128), (torch.float16, 128, 64), (torch.bfloat16, 64, 64)])
def test_kda_strong_decay(dtype, K, V):
    """One channel of the second, all channels of the last secondary chunk decay by e^-8 a token (e^-120 across the block)."""
    q, k, v, g, beta = zoo_inputs(1, 128, 2, K, V, decay="diagonal", delta=True, dtype=dtype, seed=4)
    g = g.clone()
    g[:, 16:32, :, K // 2 + 1] = -8.0
    g[:, 48:64] = -8.0
    diag.run_case(q, k, v, g, beta, sigma=0.5, rot=True, label=f"kda strong decay {dtype} K={K} V={V}")


@pytest.mark.parametrize("dtype,K,cell", [(torch.float16, 128, "gla"), (torch.bfloat16, 128, "kda"), (torch.float16, 64, "kda"), (torch.bfloat16, 64, "gla")])
def test_diagonal_blocks_against_64_bits(dtype, K, cell):
    """The A matrix inside its 16 x 16 diagonal blocks, all terms positive, so that whatever an accumulation loses adds up. The
    codes and the chunk cumsum are exact restatements; what is left is the relative error e of the sum, which shows as the share
    e 2^11 at most of fp16 results on the other side of a rounding boundary. Bound: e <= 2^-22, a weight made of two
    approximate exponentials (2^-22 each at worst, of either sign, over K channels) and six roundings of a full sum."""
    from linquant_b200.kernels import zoo

    C, H, NT, V = 64, 8, 16, 64
    gen = torch.Generator().manual_seed(11)
    u = lambda *s: torch.rand(*s, generator=gen)  # noqa: E731
    q, k = ((u(1, C * NT, H, K) * 0.5 + 0.5).to(dtype).cuda() for _ in range(2))
    v, g, beta = u(1, C * NT, H, V).to(dtype).cuda(), (-0.1 * u(1, C * NT, H, K)).cuda(), u(1, C * NT, H).cuda()
    full = lambda x, *s: torch.full(s, x, device="cuda")  # noqa: E731
    scale, sq, sk = K**-0.5, K**-0.5 / 127, 1 / 127
    sc = {"q": full(sq, H), "k": full(sk, H), "kw": full(sk, H, K), "vl": full(1 / 127, H, V), "vw": full(1 / 127, H, V), "state": full(1.0, H, V),
          "w": full(1.0, H), "el": full(1.0, H, V), "ew": full(1.0, H, V)}
    dbg = {}
    args = (q, k, v, g) + ((beta,) if cell == "kda" else ())
    getattr(zoo, f"chunk_{cell}_int8")(*args, sc, eta=0.0, _debug=dbg)
    tile = lambda x: x[0].transpose(0, 1).reshape(H * NT * 4, 16, K)  # noqa: E731
    code = lambda x, s: torch.trunc((x * (1.0 / s[0])).clamp(-127, 127) + 0.5).double()  # noqa: E731
    qc, kc = code(tile(q).float() * scale, sc["q"]), code(tile(k).float(), sc["k"])
    gc = tile(g.double().unflatten(1, (NT, C)).cumsum(2).flatten(1, 2).float()).double()
    want = torch.stack([(qc[:, i:i + 1] * kc * torch.exp(gc[:, i:i + 1] - gc)).sum(-1) for i in range(16)], 1)
    want = (want * (sc["q"][0] * sc["k"][0]).double()).tril()
    got = dbg["workspace"].view("amat").view(H * NT, 4, 16, 4, 16).diagonal(dim1=1, dim2=3).permute(0, 3, 1, 2).reshape(-1, 16, 16)
    low = torch.ones(16, 16, device="cuda").tril().bool()
    share = (got.double() != want.half().double())[:, low].double().mean().item()
    assert torch.isfinite(got).all() and (want[:, low] > 0).all() and share <= 2.0**-11, f"{share:.2e} of the fp16 results differ"
