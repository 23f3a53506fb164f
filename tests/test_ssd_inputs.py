"""Mamba-2 operands that do not fit one another: an exception on the host before the kernel that would read them."""

import pytest
import torch

B, L, H, P, G, N, C = 2, 256, 4, 64, 2, 64, 64
NC = L // C


def z(*s, dtype=torch.float32, device="cpu"):
    return torch.zeros(*s, dtype=dtype, device=device)


def i8(*s):
    return z(*s, dtype=torch.int8)


class Reached(Exception):
    pass


@pytest.fixture
def ops(monkeypatch):
    """The wrappers on CPU tensors up to the point where they would build their descriptor."""
    from linquant_b200.kernels.mamba2 import _ssd

    def call(*a, **k):
        raise Reached

    monkeypatch.setattr(_ssd, "require_cuda", lambda *a: None)
    monkeypatch.setattr(_ssd, "Call", call)


def wrappers():
    from linquant_b200.kernels.mamba2 import bmm_chunk, chunk_scan_v2, chunk_state, chunk_state_keyside, state_passing

    x, dt = z(B, L, H, P, dtype=torch.float16), z(B, H, NC, C)
    b_fp = z(B, L, G, N, dtype=torch.float16)
    return {
        "chunk_state": (chunk_state._quant_chunk_state_fwd_xfp_static_int8,
                        dict(x_fp=x, q_B=i8(B, L, G, N), dt=dt, dA_cumsum=dt, alpha_hp=z(H, P), bscale_g=z(G), out_qscale=z(H, P)),
                        ("q_B", "dt", "dA_cumsum", "bscale_g")),
        "chunk_state_keyside": (chunk_state_keyside._chunk_state_keyside_fwd,
                                dict(x_fp=x, x_scale_hp=z(H, P), b_fp=b_fp, dt=dt, dA_cumsum=dt, out_qscale=z(H, P),
                                     b_gate_scale=z(1, 1, H, N)), ("b_fp", "dt", "dA_cumsum", "b_gate_scale")),
        "bmm_chunk": (bmm_chunk._quant_bmm_chunk_fwd, dict(a=i8(B, L, G, N), a_scale=z(G), b=i8(B, L, G, N), b_scale=z(G), chunk_size=C,
                                                           static_cb_scale=z(G)), ("b", "static_cb_scale")),
        "chunk_scan": (chunk_scan_v2._quant_chunk_scan_fwd,
                       dict(cb_i8=i8(B, NC, G, C, C), x_fp=x, dt=dt, dA_cumsum=dt, q_C=i8(B, L, G, N), C_scale=z(G),
                            states=i8(B, NC, H, P, N), q_D=z(H), D_scale=1.0, state_dequant_scale=z(H, P), cb_scale=z(G)),
                       ("cb_i8", "dt", "dA_cumsum", "q_C", "states", "q_D")),
        "state_passing": (state_passing._fixedpoint_state_passing_fwd, dict(states_i8=i8(B, NC, H, P * N), dA_chunk_cumsum=dt[..., -1]),
                          ("dA_chunk_cumsum",)),
    }


@pytest.mark.parametrize("op", ["chunk_state", "chunk_state_keyside", "bmm_chunk", "chunk_scan", "state_passing"])
def test_wrappers_refuse_other_extents_and_dtypes(op, ops):
    fn, args, names = wrappers()[op]
    with pytest.raises(Reached):  # the arguments as they are pass
        fn(**args)
    for name in names:
        t = args[name]
        for axis in range(t.dim()):
            if (name, axis) in (("q_B", 3), ("b_fp", 3), ("b_fp", 2)):  # d_state and groups are read off these: the C entry judges them
                continue
            if t.size(axis) > 1:  # a size of 1 broadcasts where an axis may be coarse
                with pytest.raises(AssertionError):
                    fn(**{**args, name: t.narrow(axis, 0, t.size(axis) - 1) if t.size(axis) > 2 else t.repeat_interleave(2, axis)})
        if t.dtype == torch.int8:
            with pytest.raises(NotImplementedError):
                fn(**{**args, name: t.half()})


@pytest.mark.gpu
def test_prologues_refuse_short_constants():
    from linquant_b200.kernels.hadamard import kronecker_hadamard_fwd
    from linquant_b200.kernels.mamba2.fused_split_rotate_xBC import fused_split_rotate_quant_xBC

    xBC = z(B, L, H * P + 2 * G * N, dtype=torch.float16).cuda()
    good = [torch.ones(G, N).cuda(), torch.ones(G).cuda(), torch.ones(G).cuda()]
    fused_split_rotate_quant_xBC(xBC, good[0], H, G, N, P, good[1], good[2])
    for i in range(3):
        bad = list(good)
        bad[i] = bad[i][:1]
        with pytest.raises(AssertionError):
            fused_split_rotate_quant_xBC(xBC, bad[0], H, G, N, P, bad[1], bad[2])
    with pytest.raises(AssertionError):
        fused_split_rotate_quant_xBC(xBC, good[0], H, G, N, P, good[1], good[2], dqk_b=good[0][:1], dqk_c=good[0])
    with pytest.raises(AssertionError):
        kronecker_hadamard_fwd(z(B, L, G, N, dtype=torch.float16).cuda(), good[0][:1], G)


@pytest.mark.gpu
@pytest.mark.parametrize("keyside", [False, True])
def test_combined_refuses(keyside):
    from linquant_b200.kernels.mamba2.ssd_combined import _quant_mamba_chunk_scan_combined_fwd as fwd
    from tests.test_ssd_ops import make_case

    k = {n: t.cuda() if torch.is_tensor(t) else t for n, t in make_case(B=1, L=256, H=4, G=2, N=64, chunk=64, seed=1).items()}

    def call(**over):
        a = {**k, **over}
        return fwd(a["x"], a["dt_raw"], 1.0, a["A_log"], 1.0, a["qB"], a["sB"], a["qC"], a["sC"], 64, a["D"], 1.0,
                   static_state_scale=a["state_scale"], static_cb_scale=a["cb_scale"], alpha_hp=a["alpha"], bscale_g=a["sB"],
                   keyside=keyside, x_scale_hp=a["x_scale"], b_fp=a["Bm"], b_gate_scale=a["b_gate"])[0]

    call()
    bad = [dict(dt_raw=k["dt_raw"][:, :192]), dict(dt_raw=k["dt_raw"][:, :, :3]), dict(A_log=k["A_log"][:3]), dict(qC=k["qC"][:, :192]),
           dict(D=k["D"][:3]), dict(cb_scale=k["cb_scale"][:1])]
    bad += [dict(Bm=k["Bm"][:, :192]), dict(b_gate=k["b_gate"][:, :, :3])] if keyside else [dict(qB=k["qB"][:, :192])]
    for over in bad:
        with pytest.raises(AssertionError):
            call(**over)


def test_entries_refuse_misaligned_operands():
    """Pointers only, every one of them refused ahead of any launch: nothing is read."""
    import ctypes

    from linquant_b200 import _cabi
    from linquant_b200.kernels.mamba2._ssd import SsdProblem

    p = SsdProblem(B=B, L=L, H=H, P=P, G=G, N=N, chunk=C, x_dtype=_cabi.LQ_F16, x_stride_b=L * H * P, x_stride_t=H * P, x_stride_h=P)
    optional = ("dt_bias", "dt_scale_dev", "A_log_scale_dev", "status", "carry_in", "carry_out", "wait_flags", "post_flags")
    for name, t in SsdProblem._fields_:
        if t is ctypes.c_void_p and name not in optional:
            setattr(p, name, 4096)
    for entry, extra, name, by in (("lq_ssd_bmm_chunk", (0,), "q_C", 8), ("lq_ssd_bmm_chunk", (0,), "q_B", 1), ("lq_ssd_bmm_chunk", (1,), "b_fp", 2),
                                   ("lq_ssd_chunk_scan", (), "q_C", 8), ("lq_ssd_chunk_scan", (), "cb", 4), ("lq_ssd_chunk_scan", (), "passed", 8),
                                   ("lq_ssd_chunk_scan", (), "x", 2), ("lq_ssd_state_passing", (), "states", 4), ("lq_ssd_state_passing", (), "passed", 1),
                                   ("lq_ssd_chunk_state_value", (), "q_B", 2), ("lq_ssd_chunk_state_key", (), "b_fp", 2)):
        fn = getattr(_cabi.lib(), entry)
        fn.argtypes = [ctypes.POINTER(SsdProblem)] + [ctypes.c_int] * len(extra) + [ctypes.c_void_p]
        setattr(p, name, 4096 + by)
        assert fn(ctypes.byref(p), *extra, None) == 3, (entry, name)  # LQ_ERR_ALIGN
        setattr(p, name, 4096)
