"""Infinities in the inputs: what they reach, and only that, saturates."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk,tokens", [(64, (0, 1, 31)), (128, (5,)), (192, (6, 190)), (256, (0, 100, 255))])
def test_cumsum_with_infinite_steps(chunk, tokens):
    """An infinite dt makes its own prefix and the later ones of its chunk -inf; the earlier ones and other chunks stay as they
    are."""
    from linquant_b200.kernels.mamba2.chunk_cumsum import _quant_chunk_cumsum_fwd

    B, H, NC = 2, 5, 3
    gen = torch.Generator().manual_seed(1)
    dt = torch.rand(B, NC * chunk, H, generator=gen)
    for i, t in enumerate(tokens):
        dt[i % B, (i % NC) * chunk + t, i % H] = float("inf")
    A_log = torch.rand(H, generator=gen)
    dA, dt_out = _quant_chunk_cumsum_fwd(dt.cuda(), 1.0, A_log.cuda(), 1.0, chunk)
    x = dt.view(B, NC, chunk, H).permute(0, 3, 1, 2)
    assert torch.equal(dt_out.cpu(), x)
    want = (x * -torch.exp(A_log).view(1, H, 1, 1)).double().cumsum(-1)
    got = dA.cpu().double()
    assert torch.equal(got.isinf(), want.isinf()) and not got.isnan().any()
    torch.testing.assert_close(got, want, rtol=3e-7, atol=0.0)  # exp and two roundings in fp32


@pytest.mark.parametrize("dtype,K,rot", [(torch.bfloat16, 128, True), (torch.float16, 64, True), (torch.float16, 128, True), (torch.bfloat16, 64, False)])
def test_rescaled_rows_with_infinities(dtype, K, rot):
    """D_QK ahead of the rotation: a row with one infinity has an infinity of the Hadamard sign in every channel (codes +-127),
    opposite infinities cancel to NaN in half of them (the lower clamp), every other row keeps its codes."""
    from linquant_b200.kernels.zoo import chunk_delta_int8

    from tests.helpers import zoo_inputs

    H, V, T = 3, 64, 128
    q, k, v, g, beta = (t.cuda() for t in zoo_inputs(1, T, H, K, V, decay="scalar", delta=True, dtype=dtype, seed=2))
    full = lambda *s: torch.full(s, 0.004, device="cuda")  # noqa: E731
    sc = {"q": full(H), "k": full(H), "kw": full(H, K), "state": full(H, V), "w": full(H), "el": full(H, V), "ew": full(H, V)}
    d = torch.logspace(-0.5, 0.5, K).expand(H, K).contiguous().cuda()
    signs = torch.where(torch.rand(K, generator=torch.Generator().manual_seed(3)) < 0.5, -1.0, 1.0).cuda() if rot else None
    inf = float("inf")
    hit = {(1, 0): {5: inf}, (17, 1): {K - 1: -inf}, (66, 2): {0: inf, 9: inf}, (127, 0): {3: inf, 40: -inf}}

    def codes(q, k):
        dbg = {}
        chunk_delta_int8(q, k, v, g, beta, sc, rot=signs, dqk=d, _debug=dbg)
        return [dbg["workspace"].view(n).view(H, T, K) for n in ("qq", "kl")]

    clean = codes(q, k)
    for (t, h), at in hit.items():
        for c, x in at.items():
            q[0, t, h, c] = x
            k[0, t, h, c] = x
    hadamard = torch.ones(1, 1)
    while hadamard.shape[0] < K:
        hadamard = torch.cat([torch.cat([hadamard, hadamard], 1), torch.cat([hadamard, -hadamard], 1)])
    for got, before, x in zip(codes(q, k), clean, (q, k)):
        want = before.clone()
        for (t, h), at in hit.items():
            if rot:
                row = (x[0, t, h].double().cpu() @ hadamard.double() * signs.double().cpu())
            else:
                row = torch.where(x[0, t, h].isinf(), x[0, t, h].double(), 0.0).cpu()
            out = torch.where(row.isnan(), -127.0, row.clamp(-127, 127)).to(torch.int8).cuda()
            want[h, t] = torch.where((row.cuda().isinf() | row.cuda().isnan()), out, want[h, t])
        assert torch.equal(got, want), (got != want).nonzero()[:8]
