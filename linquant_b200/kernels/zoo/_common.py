"""Host-side plumbing shared by the zoo chunk ops: problem descriptor, launch, debug views."""

from __future__ import annotations

import ctypes as C

import torch

from ... import _cabi


def signs_of(rot, K, device):
    """Accepts a (K,) +-1 sign vector or a (K,K) signed-Hadamard matrix as built by
    ``linquant.reference.hadamard_rotation`` (reference.py:232-239: Sylvester H / sqrt(K) with the signs on the
    columns) and returns the (K,) fp32 sign vector the fused Walsh-Hadamard butterfly needs."""
    if rot is None:
        return None
    rot = torch.as_tensor(rot)
    if rot.dim() == 1:
        s = rot
    else:
        assert rot.shape == (K, K), f"rotation must be ({K},{K}) or ({K},)"
        s = torch.sign(rot[0])  # row 0 of the Sylvester matrix is all ones
        ref = _sylvester(K).to(rot.dtype).to(rot.device) / K**0.5 * s
        if not torch.allclose(ref, rot, atol=1e-3):
            raise NotImplementedError("only signed Sylvester-Hadamard rotations are fused into the prologue")
    return s.to(device=device, dtype=torch.float32).contiguous()


def _sylvester(n):
    Hm = torch.ones(1, 1, dtype=torch.float64)
    while Hm.shape[0] < n:
        Hm = torch.cat([torch.cat([Hm, Hm], 1), torch.cat([Hm, -Hm], 1)], 0)
    return Hm


def _fits(t, shape):
    """The extents of ``shape`` in order; extents of 1 may be missing or added."""
    return [n for n in t.shape if n != 1] == [n for n in shape if n != 1]


def check_inputs(q, k, v, g, beta, scales, *, decay, rot_signs=None, dqk=None, initial_state=None):
    """The kernels get bare pointers and read them with q's extents and dtype: whatever does not fit raises here."""
    assert q.dim() == 4 and k.shape == q.shape and v.dim() == 4 and v.shape[:3] == q.shape[:3], \
        f"q, k [B,T,H,K] and v [B,T,H,V] do not fit: {tuple(q.shape)}, {tuple(k.shape)}, {tuple(v.shape)}"
    if not (q.dtype == k.dtype == v.dtype):
        raise NotImplementedError(f"q, k and v must have one dtype (got {q.dtype}, {k.dtype}, {v.dtype})")
    if not (q.device == k.device == v.device):
        raise _cabi.LinQuantError(f"q, k and v must be on one device (got {q.device}, {k.device}, {v.device})")
    B, T, H, K = q.shape
    V = v.shape[3]
    want = {"g": (g, (B, T, H, K) if decay == _cabi.DECAY_DIAGONAL else (B, T, H)), "beta": (beta, (B, T, H)),
            "rot": (rot_signs, (K,)), "dqk": (dqk, (H, K)), "initial_state": (initial_state, (B, H, K, V))}
    keys = {"q": (H,), "k": (H,), "kw": (H, K), "state": (H, V)}
    keys.update({"vl": (H, V), "vw": (H, V)} if beta is None else {"w": (H,), "el": (H, V), "ew": (H, V)})
    want.update({f"scale {n!r}": (scales.get(n), shape) for n, shape in keys.items()})
    for name, (t, shape) in want.items():
        assert t is None or _fits(t, shape), f"{name} has shape {tuple(t.shape)}, {shape} expected"


def make_problem(q, k, v, g, beta, scales, *, decay, eta, sigma, tau, scale, chunk_size, bits, out, final_state,
                 rot_signs, dqk, keep, initial_state=None, unrot=None):
    """Builds the C descriptor. ``keep`` collects every temporary tensor whose storage the descriptor points to."""
    check_inputs(q, k, v, g, beta, scales, decay=decay, rot_signs=rot_signs, dqk=dqk, initial_state=initial_state)
    B, T, H, K = q.shape
    V = v.shape[-1]
    dev = q.device
    P = _cabi.ZooProblem()
    P.B, P.T, P.H, P.K, P.V, P.chunk = B, T, H, K, V, chunk_size
    P.act_dtype, P.out_dtype, P.decay = _cabi.dtype_code(q.dtype), _cabi.dtype_code(out.dtype), decay
    P.scale, P.eta, P.sigma, P.tau = float(scale), float(eta), float(sigma), float(tau)
    P.qmax = float(2 ** (bits - 1) - 1)

    def put(name, t):
        keep.append(t)
        setattr(P, name, None if t is None else t.data_ptr())

    put("q", q); put("k", k); put("v", v)
    gd = _cabi.f32c(g, dev)
    if gd is not None and decay == _cabi.DECAY_DIAGONAL and gd.data_ptr() % 16:  # read in 16-byte pieces
        gd = gd.clone()
    put("g", gd)
    put("beta", _cabi.f32c(beta, dev))
    put("rot_signs", rot_signs)
    put("dqk", _cabi.f32c(dqk, dev))
    for name, key in (("sq", "q"), ("sk", "k"), ("skw", "kw"), ("svl", "vl"), ("svw", "vw"), ("sstate", "state"),
                      ("sw", "w"), ("sel", "el"), ("sew", "ew")):
        put(name, _cabi.f32c(scales.get(key), dev))
    put("o", out)
    put("final_state", final_state)
    put("initial_state", _cabi.f32c(initial_state, dev))
    if unrot is not None:  # the kernels want the fp16 matrix with the input index contiguous: element [v'][v] = unrot[v][v']
        assert tuple(unrot.shape) == (V, V), f"unrot must be ({V},{V})"
        unrot = unrot.to(device=dev, dtype=torch.float16).t().contiguous()
    put("unrot_t", unrot)
    P.status = _cabi.status_word(dev).data_ptr()  # sticky per-device word: read by linquant_b200.check_status()
    return P


CELLS = {"lq_simple_gla_fwd": 0, "lq_gla_fwd": 1, "lq_delta_fwd": 2, "lq_kda_fwd": 3}


def call(entry, q, k, v, g, beta, scales, eta, sigma, tau, scale, chunk_size, output_final_state, unrot, bits, out_dtype, rot,
         dqk, initial_state, debug):
    """One whole-call entry on torch tensors. The native host path takes every call whose tensors are in the kernels' form
    (or need no more than an fp32 / dense copy); anything else, and a call that wants its workspace back, goes through the
    descriptor below."""
    if rot is not None and not (isinstance(rot, torch.Tensor) and rot.dim() == 1):
        rot = signs_of(rot, q.shape[-1], q.device)
    if debug is None:
        r = _cabi.host().zoo_fwd(CELLS[entry], q, k, v, g, beta, scales, eta, sigma, tau, scale, chunk_size, output_final_state,
                                 unrot, bits, out_dtype, rot, dqk, initial_state)
        if type(r) is tuple:
            return r
        if r is not None:
            _cabi.check(r, entry)
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    B, T, H, K = q.shape
    V = v.shape[-1]
    assert T % chunk_size == 0 and K <= 128, f"T={T} must be a multiple of the chunk size {chunk_size}, K={K} at most 128"
    o = torch.empty(v.shape, dtype=out_dtype or v.dtype, device=v.device)
    ht = torch.empty(B, H, K, V, dtype=torch.float32, device=q.device) if output_final_state else None
    keep = []
    decay = _cabi.DECAY_DIAGONAL if CELLS[entry] & 1 else _cabi.DECAY_NONE if g is None else _cabi.DECAY_SCALAR
    P = make_problem(q, k, v, g, beta, scales, decay=decay, eta=eta, sigma=sigma, tau=tau,
                     scale=K**-0.5 if scale is None else scale, chunk_size=chunk_size, bits=bits, out=o, final_state=ht,
                     rot_signs=signs_of(rot, K, q.device), dqk=dqk, keep=keep, unrot=unrot, initial_state=initial_state)
    run(entry, P, CELLS[entry] >= 2, q, debug)
    return o, ht


def run(entry, P, delta, like, debug=None):
    L = _cabi.lib()
    ws = _cabi.Workspace(P, delta, like.device)
    fn = getattr(L, entry)
    fn.argtypes = [C.POINTER(_cabi.ZooProblem), C.c_void_p, C.c_size_t, C.c_void_p]
    with torch.cuda.device(like.device):
        _cabi.check(fn(C.byref(P), C.c_void_p(ws.base), C.c_size_t(ws.nbytes), _cabi.stream_of(like)), entry)
    if debug is not None:
        debug["workspace"] = ws
    return ws


def run_stage(entry, P, ws, like):
    """Launch one pipeline stage (``lq_zoo_prologue_linear`` ...) on an already carved workspace."""
    L = _cabi.lib()
    fn = getattr(L, entry)
    fn.argtypes = [C.POINTER(_cabi.ZooProblem), C.POINTER(_cabi.ZooWorkspace), C.c_void_p]
    with torch.cuda.device(like.device):
        _cabi.check(fn(C.byref(P), C.byref(ws.desc), _cabi.stream_of(like)), entry)
