"""Torch-tensor front end over the C ABI, named after the reference operators.

``gated_delta_scan`` mirrors ``Program.GatedDeltaScan`` (arch/ir.go:586-603):
inputs q,k [B,T,H,Dk], v [B,T,H,Dv], beta, gate [B,T,H], IntParams
[B,T,H,Dk,Dv,chunk]; ``mamba3_selective_scan`` mirrors
``Program.Mamba3SelectiveScan`` (arch/ir.go:528-553).  Every tensor must be a
contiguous CUDA tensor; nothing here computes on the CPU.  Operand checks, result
allocation, the cached workspace and the C ABI calls are native (csrc/front.cpp).
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from ._lib import GdnDesc, Mamba3Desc, MXB_BF16, MXB_F32

_front = None


def _native():
    """The native front end, bound to the library on first use."""
    global _front
    if _front is None:
        try:
            from . import _front as module
        except ImportError as e:
            raise ImportError(f"mixlab_b200/_front.so cannot be loaded ({e}): build it with `python -m mixlab_b200.build`") from e
        _lib.lib()  # a missing library is reported the same way everywhere
        module.open(_lib.LIB_PATH)
        _front = module
    return _front


def _io(t: torch.Tensor) -> int:
    if t.dtype == torch.float32:
        return MXB_F32
    if t.dtype == torch.bfloat16:
        return MXB_BF16
    raise TypeError(f"unsupported dtype {t.dtype} (float32 or bfloat16)")


def workspace(nbytes: int, device) -> torch.Tensor:
    """The cached byte buffer of the current stream of ``device``, of at least ``nbytes`` (torch allocator).  The operators
    called on that stream use it too."""
    return _native().workspace(int(nbytes), device.index if device.index is not None else torch.cuda.current_device())


def gdn_desc(q, v, chunk, gate_is_log, flags=0) -> GdnDesc:
    B, T, H, Dk = q.shape
    return GdnDesc(B, T, H, Dk, v.shape[-1], int(chunk), _io(q), int(bool(gate_is_log)), int(flags))


def gated_delta_scan(q, k, v, beta, gate, chunk=64, *, gate_is_log=False, h0=None,
                     return_final_state=False, flags=0, save_for_backward=False):
    """Forward.  Returns out [B,T,H,Dv] (and the final state [B,H,Dk,Dv] fp32).
    ``save_for_backward`` keeps the forward intermediates in the cached workspace for a
    following ``gated_delta_scan_backward(..., use_saved=True)`` on the same inputs."""
    return (_front or _native()).gdn_forward(q, k, v, beta, gate, chunk, gate_is_log, h0, return_final_state, flags, save_for_backward)


def gated_delta_scan_backward(q, k, v, beta, gate, d_out, chunk=64, *, gate_is_log=False, h0=None,
                              d_final_state=None, flags=0, use_saved=False):
    """All gradients.  Returns dict(dq, dk, dv, dbeta, dgate, dh0)."""
    return (_front or _native()).gdn_backward(q, k, v, beta, gate, d_out, chunk, gate_is_log, h0, d_final_state, flags, use_saved)


def ir_op_forward(op_type: int, inputs, int_params, *, out_shape, float_params=()):
    """Runs one IR op record the way the reference's interpreter does after resolving its names
    (gpu/ir.cpp:4633-4654, :4837-4853): ``inputs`` in the record's order, IntParams as the Go side emits them
    (arch/ir.go:550-555, :600-602).  Returns the output tensor of ``out_shape`` in the dtype of the first input."""
    return _native().ir_op_forward(int(op_type), list(inputs), [int(v) for v in int_params], list(out_shape),
                                   [float(v) for v in float_params])


def device_status(device=None) -> int:
    """Blocking read of the device-side error word of the current stream's cached workspace (0 = ok)."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else device
    ws = workspace(256, dev)
    torch.cuda.current_stream(dev).synchronize()
    out = C.c_int32(0)
    _lib.check(_lib.lib().mxb_gdn_device_status(C.c_void_p(ws.data_ptr()), C.byref(out)), "mxb_gdn_device_status")
    return out.value


def gated_delta_decode_step(state, q, k, v, beta, gate, *, gate_is_log=False, out=None, flags=0):
    """One token on a persistent state [N,H,Dk,Dv] (updated in place).  Returns out [N,H,Dv]."""
    return (_front or _native()).gdn_decode(state, q, k, v, beta, gate, gate_is_log, out, flags)


# ---------------------------------------------------------------- gated_deltanet block stages
def gdn_block_pre(q_proj, k_proj, v_proj, conv_q, conv_k, conv_v, a_raw, b_raw, a_log, dt_bias, H, Dk, Dv, *,
                  gate_is_log=False):
    """Convolution + SiLU + L2-norm / gate / beta stage in front of the scan.  q_proj, k_proj [B,T,H*Dk],
    v_proj [B,T,H*Dv]; returns q, k [B,T,H,Dk], v [B,T,H,Dv] (I/O dtype), beta, gate [B,T,H] fp32."""
    return _native().gdn_block_pre(q_proj, k_proj, v_proj, conv_q, conv_k, conv_v, a_raw, b_raw, a_log, dt_bias, H, Dk, Dv, gate_is_log)


def gdn_block_pre_backward(q_proj, k_proj, v_proj, conv_q, conv_k, conv_v, a_raw, b_raw, a_log, dt_bias, H, Dk, Dv,
                           dq, dk, dv, dbeta, dgate, *, gate_is_log=False):
    """Gradients of gdn_block_pre: dict(dq_proj, dk_proj, dv_proj, dconv_q, dconv_k, dconv_v, da_raw, db_raw, da_log,
    ddt_bias)."""
    return _native().gdn_block_pre_backward(q_proj, k_proj, v_proj, conv_q, conv_k, conv_v, a_raw, b_raw, a_log, dt_bias, H, Dk, Dv,
                                            dq, dk, dv, dbeta, dgate, gate_is_log)


def gdn_block_post(o, z, o_norm):
    """y = RMSNorm(o, o_norm, 1e-5) * SiLU(z).  o [B,T,H,Dv], z [B,T,H*Dv] -> y [B,T,H*Dv]."""
    return _native().gdn_block_post(o, z, o_norm)


def gdn_block_post_backward(o, z, o_norm, dy):
    """Gradients of gdn_block_post: dict(do, dz, do_norm)."""
    return _native().gdn_block_post_backward(o, z, o_norm, dy)


# ---------------------------------------------------------------- Mamba-3 scan
def mamba3_desc(x, b, nheads, flags=0) -> Mamba3Desc:
    if x.dim() != 3 or b.dim() != 4:
        raise ValueError("x must be [B,T,D] and b, c [B,T,G,N]")
    B, T, D = x.shape
    G, N = b.shape[-2], b.shape[-1]
    return Mamba3Desc(B, T, D, N, G, int(nheads), _io(x), int(flags))


def mamba3_selective_scan(x, dt, lam, theta, a_log, b, c, *, nheads=0, flags=0, save_for_backward=False):
    """Forward.  x [B,T,D]; b,c [B,T,G,N]; per-channel (nheads=0) or head-broadcast parameters.
    ``save_for_backward`` keeps the chunk states in the cached workspace for a following
    ``mamba3_selective_scan_backward(..., use_saved=True)`` on the same inputs."""
    return (_front or _native()).mamba3_forward(x, dt, lam, theta, a_log, b, c, nheads, flags, save_for_backward)


def mamba3_selective_scan_backward(x, dt, lam, theta, a_log, b, c, dy, *, nheads=0, flags=0, use_saved=False):
    """Gradients in argument order.  Returns dict(dx, ddt, dlambda, dtheta, da_log, db, dc)."""
    return (_front or _native()).mamba3_backward(x, dt, lam, theta, a_log, b, c, dy, nheads, flags, use_saved)


# ---------------------------------------------------------------- Mamba-3 block stages
def mamba3_block_conv(x, w):
    """Causal depthwise convolution: x [B,T,D], w [D,K] (K <= 4; tap k multiplies x[t-k])."""
    return _native().mamba3_block_conv(x, w)


def mamba3_block_conv_backward(x, w, dy):
    return _native().mamba3_block_conv_backward(x, w, dy)


def mamba3_block_bc(b_proj, c_proj, b_scale, c_scale, b_bias, c_bias, G, N, eps=1e-5):
    """b = RMSNorm(b_proj rows of N, b_scale, eps) + b_bias, same for c.  [B,T,G*N] -> [B,T,G,N]."""
    return _native().mamba3_block_bc(b_proj, c_proj, b_scale, c_scale, b_bias, c_bias, G, N, eps)


def mamba3_block_bc_backward(b_proj, c_proj, b_scale, c_scale, db, dc, G, N, eps=1e-5):
    return _native().mamba3_block_bc_backward(b_proj, c_proj, b_scale, c_scale, db, dc, G, N, eps)


def mamba3_block_post(y, z, post_norm, eps=1e-5):
    """RMSNorm(y rows of D, post_norm, eps) * z * sigmoid(z).  y, z [B,T,D]."""
    return _native().mamba3_block_post(y, z, post_norm, eps)


def mamba3_block_post_backward(y, z, post_norm, dout, eps=1e-5):
    return _native().mamba3_block_post_backward(y, z, post_norm, dout, eps)
