"""INT8 chunk_gated_delta_rule / chunk_delta_rule (delta family, no or scalar decay) on sm_100a.

Same call as ``linquant/kernels/zoo/gated_delta_rule.py:159-203``; the device work is the C-ABI entry
``lq_delta_fwd`` (WY prologue in fp32-grade tensor-core arithmetic -> chunk-serial state pass -> output kernel)."""

from __future__ import annotations

from . import _common
from ... import _cabi


def chunk_delta_int8(q, k, v, g, beta, scales, *, sigma=1.0, tau=1.0, eta=1.0, scale=None, chunk_size=64,
                     output_final_state=False, unrot=None, fla_prep=True, bits=8, out_dtype=None, rot=None, dqk=None,
                     initial_state=None, _debug=None):
    """q,k [B,T,H,K], v [B,T,H,V] (fp16/bf16), g [B,T,H] fp32 log-decay or None (DeltaNet), beta [B,T,H].
    scales: 'q' (H,) [on q*scale], 'k' (H,) [Hw, local], 'kw' (H,K) [Hw write], 'w' (H,) [W read],
    'el' (H,V) [E local], 'ew' (H,V) [E write], 'state' (H,V).
    unrot: optional (V,V) R_V^T for canonical storage when v was rotated by R_V (the output comes out canonical).
    ``fla_prep`` is accepted for signature compatibility; the WY prep always runs in this library's own kernel.
    ``rot`` / ``dqk`` fuse the persistent R_QK rotation and the D_QK rescale into the prologue.
    Returns (o, final fp32 state [B,H,K,V] or None)."""
    if not q.is_cuda:
        raise _cabi.LinQuantError("chunk_delta_int8 runs on CUDA tensors only (no CPU path)")
    return _common.call("lq_delta_fwd", q, k, v, g, beta, scales, eta, sigma, tau, scale, chunk_size, output_final_state, unrot,
                        bits, out_dtype, rot, dqk, initial_state, _debug)
