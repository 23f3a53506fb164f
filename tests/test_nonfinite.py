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
