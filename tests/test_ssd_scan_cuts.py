"""The chunk scan where a problem is large: a call cut along the batch or the sequence gives the same bits as the whole one, whatever the
sizes on the two sides of the cut; the time does not depend on how fast the heads forget; an overflow of x is not hidden; and the
values against 64 bits, chunk by chunk, over slow and fast decays, resets and steps so large that nothing survives them."""

import pytest
import torch

pytestmark = pytest.mark.gpu
SIZE = 4096  # head-tokens per SM that the large side of every comparison has, and the small side has not


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def make(B, NC, H, G, N, C, dtype, decay, seed, D_dims=1):
    g = torch.Generator("cuda").manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    L = NC * C
    dt = torch.nn.functional.softplus(randn(B, H, NC, C) * 0.5 - 2.0)
    lo, hi = {"slow": (0.1, 3.0), "mixed": (1.0, 16.0), "fast": (40.0, 80.0), "reset": (0.5, 4.0), "wander": (0.1, 0.4)}[decay]
    if decay == "reset":  # a token in a hundred forgets everything before it
        dt = torch.where(rand(*dt.shape) < 0.01, torch.full_like(dt, 200.0), dt)
    if decay == "wander":  # log-decays that rise and fall
        dt = dt * randn(*dt.shape)
    dA = (-torch.linspace(lo, hi, H, device="cuda", dtype=torch.float64).view(1, H, 1, 1) * dt).cumsum(-1).float()
    i8 = lambda *s: torch.randint(-127, 128, s, generator=g, device="cuda", dtype=torch.int32).to(torch.int8)  # noqa: E731
    sc = lambda *s: rand(*s) * 0.01 + 0.01  # noqa: E731
    return dict(cb=i8(B, NC, G, C, C), x=randn(B, L, H, 64).to(dtype), dt=dt, dA=dA, qC=i8(B, L, G, N), sC=sc(G), passed=i8(B, NC, H, 64, N),
                D=(None, randn(H), randn(H, 64))[D_dims], sS=sc(H, 64), sCB=sc(G))


def scan(k):
    import linquant_b200
    from linquant_b200.kernels.mamba2 import ssd_combined as sc

    out = sc._chunk_scan_v2(k["cb"], k["x"], k["dt"], k["dA"], k["qC"], k["sC"], k["passed"], k["D"], torch.ones(1, device="cuda"), k["sS"], k["sCB"])
    linquant_b200.check_status("cuda")
    return out


def exact(k):
    B, L, H, P = k["x"].shape
    NC, C = k["dt"].shape[2:]
    G = k["sC"].numel()
    out = torch.empty(B, L, H, P, dtype=torch.float64, device="cuda")
    for h in range(H):
        gr = h * G // H
        X, dA = k["x"][:, :, h].double().view(B, NC, C, P), k["dA"][:, h].double()
        M = k["cb"][:, :, gr].double() * (dA.unsqueeze(-1) - dA.unsqueeze(-2)).exp().tril() * (k["sCB"][gr].double() * k["dt"][:, h].double()).unsqueeze(-2)
        read = k["qC"][:, :, gr].double().view(B, NC, C, -1) @ k["passed"][:, :, h].double().transpose(-1, -2)
        y = M @ X + read * (k["sC"][gr].double() * k["sS"][h].double()) * dA.exp().unsqueeze(-1)
        if k["D"] is not None:
            y = y + X * k["D"][h].double()
        out[:, :, h] = y.reshape(B, L, P)
    return out


@pytest.mark.parametrize("B,NC,H,G,N,C,dtype", [(2, 16, 80, 1, 128, 256, torch.bfloat16), (2, 28, 96, 2, 128, 128, torch.float16),
                                                (2, 64, 80, 2, 64, 64, torch.float16), (2, 22, 80, 1, 64, 192, torch.bfloat16)])
def test_cuts_of_batch_and_sequence_keep_every_bit(B, NC, H, G, N, C, dtype):
    from linquant_b200.kernels.mamba2 import ssd_combined as sc
    from linquant_b200.seqpar import ssd_segmented_on_one_device

    L = NC * C
    assert B * L * H >= SIZE * sms() > B * L * H // 2, "the whole call and its halves must lie on the two sides"
    g = torch.Generator("cuda").manual_seed(11)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    i8 = lambda *s: torch.randint(-127, 128, s, generator=g, device="cuda", dtype=torch.int32).to(torch.int8)  # noqa: E731
    x = torch.randn(B, L, H, 64, generator=g, device="cuda").to(dtype)
    dt = torch.randn(B, L, H, generator=g, device="cuda") * 0.5 - 2.0
    qB, qC, sB, sC = i8(B, L, G, N), i8(B, L, G, N), rand(G) * 0.01 + 0.01, rand(G) * 0.01 + 0.01
    A_log, D = rand(H) * 2.7, torch.randn(H, generator=g, device="cuda")
    kw = dict(dt_softplus=True, static_state_scale=rand(H, 64) * 0.1 + 0.1, static_cb_scale=rand(G) * 0.1 + 0.1, alpha_hp=rand(H, 64) * 0.01 + 0.01,
              bscale_g=sB)
    fwd = lambda s: sc._quant_mamba_chunk_scan_combined_fwd(  # noqa: E731
        x[s], dt[s], 1.0, A_log, 1.0, qB[s], sB, qC[s], sC, C, D, 1.0, **kw)[0]
    whole = fwd(slice(None))
    for b in range(B):
        assert torch.equal(fwd(slice(b, b + 1)), whole[b:b + 1]), f"batch element {b} alone differs from its rows of the whole call"
    seg = ssd_segmented_on_one_device(2, x, dt, 1.0, A_log, 1.0, qB, sB, qC, sC, C, D, 1.0, **kw)
    assert torch.equal(seg, whole), "two chained segments differ from the single call"


@pytest.mark.parametrize("C,N", [(256, 128), (64, 64)])
def test_time_does_not_depend_on_the_decay(C, N):
    """A serving call meets heads of every decay: twice the time of slow heads is far outside the scatter of a kernel that does the same
    work for all of them."""
    times = {}
    for decay in ("slow", "fast", "reset"):
        k = make(2, 4096 // C, 80, 1, N, C, torch.bfloat16, decay, 4)
        assert k["x"].numel() // 64 >= SIZE * sms()
        best = float("inf")
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            scan(k)
            e0.record()
            scan(k)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        times[decay] = best
    assert max(times.values()) < 2 * times["slow"], times


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C,N", [(256, 128), (64, 64)])
def test_opposite_infinities_reach_every_later_row(C, N, dtype):
    """inf - inf and 0 * inf are NaN: equal codes for the two tokens, or a zero code, must not make a later row finite."""
    k = make(1, 20480 // C, 32, 1, N, C, dtype, "slow", 7)
    assert k["x"].numel() // 64 >= SIZE * sms()
    k["cb"][0, 0, 0, :, 20] = 1
    k["cb"][0, 0, 0, :, 30] = 1
    k["cb"][0, 0, 0, C - 4:, 20:31] = 0
    k["x"][0, 20, 0, 5], k["x"][0, 30, 0, 5] = float("inf"), float("-inf")
    assert not torch.isfinite(scan(k)[0, 30:C, 0, 5]).any()


def check(o, k, e):
    """Relative error of each (batch, chunk, head) by itself, so that rows with large steps do not outweigh the rest. A weight is rounded
    to fp16 up to three times (relative 2^-11 each, once more for D on the diagonal) and the output once: 5 * 2^-11 = 2.4e-3 if every
    rounding were at its bound with the same sign."""
    B, L, H, P = o.shape
    NC, C = k["dt"].shape[2:]
    o, e = o.double().view(B, NC, C, H, P), e.view(B, NC, C, H, P)
    err = (o - e).pow(2).sum((2, 4)).sqrt() / e.pow(2).sum((2, 4)).sqrt()
    assert float(err.max()) < 2.4e-3, f"worst chunk {float(err.max()):.2e}, mean {float(err.mean()):.2e}"


@pytest.mark.parametrize("decay", ["slow", "mixed", "fast", "reset", "wander"])
@pytest.mark.parametrize("B,NC,H,G,N,C,dtype,D_dims", [(2, 80, 16, 1, 128, 256, torch.bfloat16, 1), (2, 80, 16, 2, 64, 256, torch.float16, 2),
                                                       (2, 106, 16, 2, 128, 192, torch.bfloat16, 0), (1, 291, 33, 1, 64, 64, torch.bfloat16, 2),
                                                       (1, 101, 7, 7, 128, 128, torch.float16, 1), (1, 1, 1, 1, 128, 256, torch.bfloat16, 2),
                                                       (1, 5, 3, 1, 64, 192, torch.bfloat16, 1)])
def test_every_chunk_against_64_bits(B, NC, H, G, N, C, dtype, D_dims, decay):
    k = make(B, NC, H, G, N, C, dtype, decay, 3, D_dims)
    check(scan(k), k, exact(k))


@pytest.mark.parametrize("H,NC,C,N", [(1, 2399, 256, 128), (149, 33, 128, 128), (37, 65, 256, 64), (33, 291, 64, 128), (7, 500, 192, 64)])
def test_item_counts_that_do_not_divide_among_the_sms(H, NC, C, N):
    k = make(1, NC, H, 1, N, C, torch.bfloat16, "mixed", 5)
    check(scan(k), k, exact(k))


def test_x_as_a_view_into_wider_rows():
    k = make(2, 40, 32, 1, 128, 256, torch.bfloat16, "mixed", 6)
    wide = torch.full((2, k["x"].shape[1], 32 * 64 + 256), 7.0, device="cuda", dtype=torch.bfloat16)
    wide[..., :2048] = k["x"].flatten(-2)
    e = exact(k)
    k["x"] = wide[..., :2048].unflatten(-1, (32, 64))
    check(scan(k), k, e)
