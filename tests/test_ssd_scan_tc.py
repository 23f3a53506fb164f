"""The chunk scan with its codes in tensor memory against 64 bits, at the decays where its split of the decay changes: one segment over
the whole chunk, a segment per row block or less, rows that forget so fast that they are summed one by one, steps that reset the
state. Every case has the 4096 head-tokens per SM from which the kernel is the library's choice."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def make(B, NC, H, G, N, C, dtype, decay, seed, dmode):
    assert B * NC * C * H >= 4096 * torch.cuda.get_device_properties(0).multi_processor_count, "too small for the kernel under test"
    g = torch.Generator("cuda").manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    L = NC * C
    dt = torch.nn.functional.softplus(randn(B, H, NC, C) * 0.5 - 2.0)
    lo, hi = {"slow": (0.1, 3.0), "mixed": (1.0, 16.0), "fast": (40.0, 80.0), "reset": (0.5, 4.0), "wander": (0.1, 0.4)}[decay]
    A = torch.linspace(lo, hi, H, device="cuda").view(1, H, 1, 1)
    if decay == "reset":  # a token in a hundred forgets everything before it
        dt = torch.where(rand(*dt.shape) < 0.01, torch.full_like(dt, 200.0), dt)
    if decay == "wander":  # log-decays that rise and fall
        dt = dt * randn(*dt.shape)
    dA = (-A.double() * dt.double()).cumsum(-1).float()
    i8 = lambda *s: torch.randint(-127, 128, s, generator=g, device="cuda").to(torch.int8)  # noqa: E731
    sc = lambda *s: rand(*s) * 0.01 + 0.01  # noqa: E731
    D = None if dmode == 0 else randn(H) if dmode == 1 else randn(H, 64)
    return dict(cb=i8(B, NC, G, C, C), x=randn(B, L, H, 64).to(dtype), dt=dt, dA=dA, qC=i8(B, L, G, N), sC=sc(G), passed=i8(B, NC, H, 64, N),
                D=D, sS=sc(H, 64), sCB=sc(G))


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


def run(k):
    import linquant_b200
    from linquant_b200.kernels.mamba2 import ssd_combined as sc

    out = sc._chunk_scan_v2(k["cb"], k["x"], k["dt"], k["dA"], k["qC"], k["sC"], k["passed"], k["D"], torch.ones(1, device="cuda"), k["sS"], k["sCB"])
    linquant_b200.check_status("cuda")
    return out


def check(o, e):
    """Rounding the output to fp16 alone is a relative error of 2.1e-4 (2^-11 / sqrt(12) over a mantissa); the pieces (2^-17) and the
    exponentials (1e-5) add nothing to it that would show. One element: half a step of fp16, 2^-11 of the largest value."""
    err = float((o.double() - e).norm() / e.norm())
    assert err < 2.5e-4, f"relative error {err:.2e}"
    assert float((o.double() - e).abs().max() / e.abs().max()) < 6e-4


@pytest.mark.parametrize("decay", ["slow", "mixed", "fast", "reset", "wander"])
@pytest.mark.parametrize("C,N,dtype,G,dmode", [(256, 128, torch.bfloat16, 1, 1), (256, 64, torch.float16, 2, 2), (192, 128, torch.bfloat16, 2, 0),
                                               (128, 128, torch.float16, 1, 1), (64, 64, torch.bfloat16, 1, 2)])
def test_scan_against_64_bits(C, N, dtype, G, dmode, decay):
    k = make(2, 80 * 256 // C, 16, G, N, C, dtype, decay, 3, dmode)
    check(run(k), exact(k))


@pytest.mark.parametrize("H,NC,C,N", [(1, 2399, 256, 128), (149, 33, 128, 128), (37, 65, 256, 64), (33, 291, 64, 128), (7, 500, 192, 64)])
def test_scan_item_counts(H, NC, C, N):
    """Items that do not divide among the SMs: a chunk per item (the codes change every time), chunks that two blocks share."""
    k = make(1, NC, H, 1, N, C, torch.bfloat16, "mixed", 5, 1)
    check(run(k), exact(k))


def test_scan_of_a_strided_view():
    """x as a view into a wider row, batch stride and all."""
    k = make(2, 40, 32, 1, 128, 256, torch.bfloat16, "mixed", 6, 1)
    wide = torch.full((2, k["x"].shape[1], 32 * 64 + 256), 7.0, device="cuda", dtype=torch.bfloat16)
    wide[..., :2048] = k["x"].flatten(-2)
    e = exact(k)
    k["x"] = wide[..., :2048].unflatten(-1, (32, 64))
    check(run(k), e)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_scan_infinite_value_reaches_later_rows_only(dtype):
    k = make(1, 80, 32, 1, 128, 256, dtype, "slow", 7, 1)
    k["cb"][k["cb"] == 0] = 1
    e = exact(k)
    k["x"][0, 70, 0, 5] = float("inf")
    o = run(k)
    hit = torch.zeros(o.shape, dtype=torch.bool, device="cuda")
    hit[0, 70:256, 0, 5] = True
    assert not torch.isfinite(o[hit]).any()
    check(o[~hit], e[~hit])
