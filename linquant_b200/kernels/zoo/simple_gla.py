"""INT8 chunk_simple_gla (linear attention with no or scalar decay) on sm_100a.

Same call as ``linquant/kernels/zoo/simple_gla.py:175-212``; the device work is the C-ABI entry
``lq_simple_gla_fwd`` (fused prologue -> tiled state pass -> output kernel)."""

from __future__ import annotations

from . import _common
from ... import _cabi


def chunk_simple_gla_int8(q, k, v, g, scales, *, eta=1.0, scale=None, chunk_size=64, output_final_state=False,
                          unrot=None, bits=8, out_dtype=None, rot=None, dqk=None, initial_state=None, _debug=None):
    """q,k [B,T,H,K], v [B,T,H,V] (fp16/bf16), g [B,T,H] fp32 log-decay or None.
    scales: dict with 'q' (H,) [calibrated on q*scale], 'k' (H,), 'kw' (H,K), 'vw' (H,V), 'vl' (H,V), 'state' (H,V),
    fp32 on q's device. T must be a multiple of chunk_size.
    unrot: optional (V,V) R_V^T for canonical storage when v was rotated by R_V (the output comes out canonical).
    Extensions over the reference signature (all optional): ``rot`` fuses the persistent signed-Hadamard R_QK into
    the prologue (a (K,) sign vector or the (K,K) matrix of ``hadamard_rotation``); ``dqk`` (H,K) fuses the
    diagonal rescale q*D, k/D ahead of it; ``initial_state`` (B,H,K,V) fp32 is the carry entering the first chunk
    (zero when omitted), which is what a sequence split over several calls or GPUs hands from one segment to the next.
    Returns (o [B,T,H,V] in v.dtype or out_dtype, final fp32 state [B,H,K,V] or None)."""
    if not q.is_cuda:
        raise _cabi.LinQuantError("chunk_simple_gla_int8 runs on CUDA tensors only (no CPU path)")
    return _common.call("lq_simple_gla_fwd", q, k, v, g, None, scales, eta, 1.0, 1.0, scale, chunk_size, output_final_state, unrot,
                        bits, out_dtype, rot, dqk, initial_state, _debug)
