"""Performance cases of the INT8 chunk-prefill path, through the calls a serving program makes.

Two families of operations:

* ``zoo`` -- one attention layer's chunk call (simple GLA, GLA, DeltaNet / Gated DeltaNet, KDA) with the rotation fused
  into the call, static scales calibrated beforehand on other data of the same distribution;
* ``ssd`` -- one Mamba-2 mixer's SSD region: the split / rotate / quantise prologue on xBC, then the combined forward, with
  value-side or key-side absorption.

Sizes span a short prompt of one user up to the full-size benchmark configurations. The path is prefill only: it has no
backward pass and no single-token decode, and every length is a multiple of the chunk size."""

import math

import torch
import torch.nn.functional as F

from linquant_b200 import invariances as inv
from linquant_b200.kernels.hadamard import kronecker_hadamard_fwd
from linquant_b200.kernels.mamba2.calibration import SsdObservers
from linquant_b200.kernels.mamba2.fused_split_rotate_xBC import fused_split_rotate_quant_xBC
from linquant_b200.kernels.mamba2.ssd_combined import _quant_mamba_chunk_scan_combined_fwd
from linquant_b200.kernels.zoo import chunk_delta_int8, chunk_gla_int8, chunk_kda_int8, chunk_simple_gla_int8

CHUNK = 64  # of the zoo operations
HEADDIM = 64  # of the SSD operations
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def _zoo(op, B, T, H, K=128, V=128, dtype="bf16", policy="kernel_static", decay="scalar", eta=1.0, sigma=1.0, tau=1.0,
         dqk=False, resume=False):
    """``resume``: the call continues a cached prefix (a carry comes in) and hands its own carry on."""
    return dict(family="zoo", op=op, B=B, T=T, H=H, K=K, V=V, dtype=dtype, policy=policy, decay=decay, eta=eta, sigma=sigma,
                tau=tau, dqk=dqk, resume=resume)


def _ssd(B, L, H, N=128, G=1, chunk=256, dtype="bf16", keyside=False):
    return dict(family="ssd", B=B, L=L, H=H, N=N, G=G, chunk=chunk, dtype=dtype, keyside=keyside)


def listed():
    cases = {
        # simple GLA: a one-user prompt of 128 tokens, where latency and launches are the cost
        "simple_gla_prompt": _zoo("simple_gla", 1, 128, 16, policy="kernel_pt"),
        # simple GLA: the full benchmark configuration (a batch of four 4096-token prompts)
        "simple_gla_batch": _zoo("simple_gla", 4, 4096, 16, policy="kernel_pt"),
        # linear attention on 64-channel heads in fp16, an odd number of heads and chunks, continuing a cached prefix
        "simple_gla_resume_f16": _zoo("simple_gla", 3, 37 * CHUNK, 5, 64, 64, dtype="f16", eta=0.5, resume=True),
        # GLA: per-channel decay, two long prompts
        "gla_batch": _zoo("gla", 2, 4096, 16, decay="diagonal", eta=0.0),
        # DeltaNet without decay: one prompt, fp16
        "deltanet_prompt_f16": _zoo("delta", 1, 1024, 16, dtype="f16", decay="none"),
        # Gated DeltaNet: the full benchmark configuration, with the diagonal query / key rescale
        "gated_deltanet_batch": _zoo("delta", 4, 8192, 16, policy="kernel_ptk", sigma=0.5, dqk=True),
        # KDA: one prompt of a ragged number of chunks
        "kda_prompt": _zoo("kda", 1, 31 * CHUNK, 32, decay="diagonal", eta=0.0),
        # KDA: the full benchmark configuration, the most expensive call of the library
        "kda_batch": _zoo("kda", 8, 8192, 32, decay="diagonal", eta=0.0),
        # Mamba-2 2.7B-shaped mixer: a one-user prompt of a single 256-token chunk
        "mamba2_prompt": _ssd(1, 256, 80),
        # Mamba-2 2.7B-shaped mixer: the full benchmark configuration
        "mamba2_batch": _ssd(8, 16384, 80),
        # the same mixer with key-side absorption on two 4096-token prompts
        "mamba2_keyside": _ssd(2, 4096, 80, keyside=True),
        # a smaller mixer: d_state 64, chunk 64, two groups, fp16, an odd number of chunks
        "mamba2_n64_f16": _ssd(3, 33 * 64, 24, N=64, G=2, chunk=64, dtype="f16"),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """Lengths are log-uniform from one chunk to 16384 tokens; the batch keeps the call within the largest listed one."""
    dtype = rng.choice(("bf16", "bf16", "f16"))
    if rng.random() < 0.4:
        G = rng.choice((1, 1, 2))
        H = G * _log_int(rng, 4, 80 // G)
        N = rng.choice((128, 128, 64))
        chunk = rng.choice((256, 256, 128, 192, 64))
        L = chunk * _log_int(rng, 1, 16384 // chunk)
        B = _log_int(rng, 1, max(1, min(8, 10_485_760 // (L * H))))
        return _ssd(B, L, H, N, G, chunk, dtype, rng.random() < 0.3)
    op = rng.choice(("simple_gla", "gla", "delta", "kda"))
    K, V = rng.choice(((128, 128), (128, 128), (64, 64), (128, 64), (64, 128)))
    H = _log_int(rng, 1, 32)
    T = CHUNK * _log_int(rng, 1, 256)
    most = 2_097_152 if op == "kda" else 1_048_576  # head-tokens
    B = _log_int(rng, 1, max(1, min(8, most // (T * H))))
    diagonal = op in ("gla", "kda")
    return _zoo(op, B, T, H, K, V, dtype, rng.choice(("kernel_static", "kernel_pt", "kernel_ptk")),
                "diagonal" if diagonal else rng.choice(("scalar", "scalar", "none")),
                rng.choice((0.0, 0.5)) if diagonal else rng.choice((1.0, 1.0, 0.5)),
                rng.choice((1.0, 0.5)) if op in ("delta", "kda") else 1.0, 1.0,
                not diagonal and rng.random() < 0.25, rng.random() < 0.25)


# ---------------------------------------------------------------------------------------------------------- inputs
def _zoo_inputs(c, gen, B, T):
    """The distributions of the benchmark configurations: unit-norm keys (heavy channels for KDA), unit-norm queries for
    the delta rule, log-sigmoid gates, sigmoid write strengths."""
    dev, dt = "cuda", DTYPES[c["dtype"]]
    H, K, V = c["H"], c["K"], c["V"]
    heavy = torch.randperm(K, generator=gen, device=dev)[: max(1, round(0.01 * K))]
    out = {n: [] for n in ("q", "k", "v", "g", "beta")}
    for _ in range(B):
        q = torch.randn(T, H, K, generator=gen, device=dev)
        k = torch.randn(T, H, K, generator=gen, device=dev)
        if c["op"] == "delta":
            q = F.normalize(q, dim=-1)
        if c["op"] == "kda":
            k[..., heavy] *= 20.0
        out["q"].append(q.to(dt))
        out["k"].append(F.normalize(k, dim=-1).to(dt))
        out["v"].append(torch.randn(T, H, V, generator=gen, device=dev).to(dt))
        if c["decay"] != "none":
            shape = (T, H, K) if c["decay"] == "diagonal" else (T, H)
            mean = 4.0 if c["op"] == "kda" else 3.0
            out["g"].append(F.logsigmoid(torch.randn(*shape, generator=gen, device=dev) + mean))
        if c["op"] in ("delta", "kda"):
            out["beta"].append(torch.sigmoid(torch.randn(T, H, generator=gen, device=dev)))
    return {n: torch.stack(v) if v else None for n, v in out.items()}


def _prepare_zoo(c, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    B, T, H, K, V = c["B"], c["T"], c["H"], c["K"], c["V"]
    signs = inv.hadamard_signs(K, 0).cuda()
    # static scales from another draw of the same distribution; without a decay the state grows with the length
    cal = _zoo_inputs(c, gen, 1, min(T, 4096 if c["decay"] == "none" else 1024))
    dqk = inv.dqk_from_stats(cal["q"], cal["k"], 0.5) if c["dqk"] else None
    sc = inv.StaticScales(c["policy"])
    if c["decay"] == "diagonal":
        inv.calibrate_diagonal(sc, cal["q"], cal["k"], cal["v"], cal["g"], cal["beta"], eta=c["eta"], sigma=c["sigma"],
                               tau=c["tau"], rot_signs=signs)
    elif c["op"] == "delta":
        inv.calibrate_delta(sc, cal["q"], cal["k"], cal["v"], cal["g"], cal["beta"], eta=c["eta"], sigma=c["sigma"],
                            tau=c["tau"], rot_signs=signs, dqk=dqk)
    else:
        inv.calibrate_linear(sc, cal["q"], cal["k"], cal["v"], cal["g"], eta=c["eta"], rot_signs=signs, dqk=dqk)
    scales = sc.finalize().kernel_scales(H, K, V, "cuda")
    x = _zoo_inputs(c, gen, B, T)
    kw = dict(eta=c["eta"], rot=signs, output_final_state=c["resume"])
    if c["resume"]:
        kw["initial_state"] = torch.randn(B, H, K, V, generator=gen, device="cuda") * (30.0 * scales["state"].view(1, H, 1, V))
    if c["dqk"]:
        kw["dqk"] = dqk
    args = [x["q"], x["k"], x["v"], x["g"]]
    if c["op"] in ("delta", "kda"):
        args.append(x["beta"])
        kw.update(sigma=c["sigma"], tau=c["tau"])
    return dict(op=c["op"], args=args, scales=scales, kw=kw)


def _ssd_inputs(c, gen, heavy, B, L):
    """Post-convolution xBC ~ N(0,1) with 1 % heavy channels (x20), raw dt ~ N(-2, 0.5) ahead of its softplus."""
    width = c["H"] * HEADDIM + 2 * c["G"] * c["N"]
    xBC = torch.empty(B, L, width, dtype=DTYPES[c["dtype"]], device="cuda")
    for b in range(B):
        t = torch.randn(L, width, generator=gen, device="cuda")
        t[:, heavy] *= 20.0
        xBC[b] = t
    return xBC, torch.randn(B, L, c["H"], generator=gen, device="cuda") * 0.5 - 2.0


def _prepare_ssd(c, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    B, L, H, N, G, C = c["B"], c["L"], c["H"], c["N"], c["G"], c["chunk"]
    d_ssm, width = H * HEADDIM, H * HEADDIM + 2 * G * N
    A_log = torch.rand(H, generator=gen, device="cuda") * math.log(16.0)
    D = torch.randn(H, generator=gen, device="cuda")
    signs = torch.randint(0, 2, (G, N), generator=gen, device="cuda").float() * 2 - 1
    heavy = torch.randperm(width, generator=gen, device="cuda")[: max(1, round(0.01 * width))]
    Lc = min(L, max(1, 768 // C) * C)
    xBC, dt = _ssd_inputs(c, gen, heavy, 1, Lc)
    rot = [kronecker_hadamard_fwd(t.unflatten(-1, (G, N)).contiguous(), signs, G) for t in xBC[..., d_ssm:].split(G * N, -1)]
    scales = SsdObservers().observe(xBC[..., :d_ssm].unflatten(-1, (H, HEADDIM)), dt, A_log, *rot, C).scales()
    scales = {k: v.contiguous() for k, v in scales.items()}
    xBC, dt = _ssd_inputs(c, gen, heavy, B, L)
    return dict(op="ssd", H=H, N=N, G=G, chunk=C, keyside=c["keyside"], xBC=xBC, dt=dt, A_log=A_log, D=D, signs=signs,
                scales=scales, B_inv=1.0 / scales["B_scale"], C_inv=1.0 / scales["C_scale"])


def prepare(case, seed):
    return _prepare_ssd(case, seed) if case["family"] == "ssd" else _prepare_zoo(case, seed)


# ------------------------------------------------------------------------------------------------------- the calls
ZOO = {"simple_gla": chunk_simple_gla_int8, "gla": chunk_gla_int8, "delta": chunk_delta_int8, "kda": chunk_kda_int8}


def run(s):
    if s["op"] != "ssd":
        o, state = ZOO[s["op"]](*s["args"], s["scales"], **s["kw"])
        return {"o": o, "state": state}
    S, d_ssm, gn = s["scales"], s["H"] * HEADDIM, s["G"] * s["N"]
    x, qB, qC = fused_split_rotate_quant_xBC(s["xBC"], s["signs"], s["H"], s["G"], s["N"], HEADDIM, s["B_inv"], s["C_inv"])
    side = {}
    if s["keyside"]:  # the gate-weighted B is quantised inside the chunk state: it takes the rotated floating-point B
        b_fp = kronecker_hadamard_fwd(s["xBC"][..., d_ssm:d_ssm + gn].unflatten(-1, (s["G"], s["N"])), s["signs"], s["G"])
        side = dict(keyside=True, x_scale_hp=S["x_scale_hp"], b_fp=b_fp, b_gate_scale=S["b_gate_scale"])
    return _quant_mamba_chunk_scan_combined_fwd(
        x, s["dt"], 1.0, s["A_log"], 1.0, qB, S["B_scale"], qC, S["C_scale"], s["chunk"], s["D"], 1.0, dt_softplus=True,
        static_state_scale=S["state_scale"], static_cb_scale=S["cb_scale"], alpha_hp=S["alpha_hp"], bscale_g=S["B_scale"],
        **side)[0]


# ------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    if c["family"] == "ssd":
        ht = c["B"] * c["L"] * c["H"]
        lanes = c["G"] * c["N"] / c["H"]  # B and C lanes, shared by the heads of a group
        return {"bytes": ht * (2 * HEADDIM + 2 * HEADDIM + 4 + 2 * 2 * lanes),  # x in, out, dt, B and C
                # state write and state read, causal product, C.B^T once per group
                "flops": ht * (4 * HEADDIM * c["N"] + c["chunk"] * HEADDIM + c["chunk"] * lanes)}
    K, V, ht = c["K"], c["V"], c["B"] * c["T"] * c["H"]
    byte = 2 * (2 * K + 2 * V) + {"none": 0, "scalar": 4, "diagonal": 4 * K}[c["decay"]]
    flop = 4 * K * V + CHUNK * (K + V) + 2 * K * math.log2(K)  # state write and read, causal local product, rotation
    if c["op"] in ("delta", "kda"):
        byte += 4
        flop += 2 * K * V + CHUNK * (2 * K + V)  # state read of W, Gram matrix, W and U
    state = (2 if c["resume"] else 0) * 4 * c["B"] * c["H"] * K * V
    return {"bytes": ht * byte + state, "flops": ht * flop}


def tolerance(case):
    """Operands are INT8 codes: two correct implementations differ where an fp32 product lies on a rounding boundary (one
    step of one code in some 1e5), which moves an output by well under its fp16 / bf16 rounding. The delta rule without
    decay never forgets such a step: there the difference is of the order of the codes' own rounding."""
    if case["family"] == "zoo" and case["op"] == "delta" and case["decay"] == "none":
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 5e-3 if case["dtype"] == "bf16" else 3e-3, "max": 0.1}
