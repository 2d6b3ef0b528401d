"""Input prologue: token-major projections -> the operator's head-major inputs, in one CUDA pass each way.

The reference's driver does it with transposes and views (``main.py:24-31``); its harness additionally normalises the
keys and passes the gates through a sigmoid (``Universal_Attention/triton/_debug.py:470-475``).  ``prepare_inputs`` does
all of it in ``ua_prepare_inputs`` and is differentiable (``ua_prepare_inputs_bwd``)."""
from __future__ import annotations

from torch.autograd import Function

from . import _lib
from .universal_attention_autograd import _transforms_active


class _PrepareInputs(Function):
    @staticmethod
    def forward(ctx, query_state, key_state, value_state, gate_state, chunk, flags):
        *outs, knorm = _lib.native().prepare_inputs(query_state, key_state, value_state, gate_state, chunk, flags)
        ctx.args = (query_state.shape[2], flags)
        ctx.in_shapes = (query_state.shape, key_state.shape, value_state.shape, gate_state.shape)
        ctx.set_materialize_grads(False)                  # an output without a gradient: zeros are made natively
        ctx.save_for_backward(outs[0], outs[3], outs[4], knorm)
        return tuple(outs)

    @staticmethod
    def backward(ctx, g_kc, g_vc, g_xq, g_src, g_dest):
        kc, ssrc, sdest, knorm = ctx.saved_tensors
        n, flags = ctx.args
        grads = _lib.native().prepare_inputs_bwd(g_kc, g_vc, g_xq, g_src, g_dest, kc, ssrc, sdest, knorm, n, flags)
        return (*(g.view(s) for g, s in zip(grads, ctx.in_shapes)), None, None)


def prepare_inputs(query_state, key_state, value_state, gate_state, chunk=128, normalize_keys=False, sigmoid_gates=False):
    """``query_state (b,s,n,d)``, ``key_state, value_state (b,s,n_kv,d)``, ``gate_state (b,s,2*n_kv)`` (source gates
    first, as ``main.py:29-31`` splits them) -> ``(kc, vc, xq, static_src, static_dest)`` in the operator's 1-D layout:
    ``kc, vc (b,n_kv,s/chunk,chunk,d)``, ``xq (b,n_kv,n/n_kv,s,d)``, ``static_src (b,n_kv,s/chunk,chunk)``,
    ``static_dest (b,n_kv,s)``.  ``normalize_keys``: keys divided by ``|k| + 1e-6``; ``sigmoid_gates``: gates =
    sigmoid(gate_state).  Differentiable with respect to the four projections."""
    flags = (_lib.PREP_NORMALIZE_KEYS if normalize_keys else 0) | (_lib.PREP_SIGMOID_GATES if sigmoid_gates else 0)
    apply = _PrepareInputs.apply if _transforms_active() else _lib.native().prepare_apply
    return apply(query_state, key_state, value_state, gate_state, chunk, flags)
