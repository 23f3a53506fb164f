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
