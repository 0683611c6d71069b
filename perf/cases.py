"""The work a user has this framework do, as measurable cases.

Kinds of work, all through the public entry points (``mixlab_b200.ops`` and, for host buffers, the C ABI):

  decode        one token of the gated delta recurrence on a persistent state (serving)
  scan          the gated delta scan: forward alone (prefill, evaluation) or forward + backward (training)
  gdn_layer     one gated_deltanet layer without its matrix products: convolution / norm / gate stage, scan, output stage,
                forward and every gradient
  mamba3        the Mamba-3 selective scan, forward alone or forward + backward
  mamba3_layer  one canonical Mamba-3 layer without its matrix products, forward and every gradient
  host          the gated delta scan on host buffers (what the cgo bridge calls), forward + backward

``listed()`` names a dozen of them, ``draw()`` gives others of the same ranges.
"""
import ctypes
import math

import torch
import torch.nn.functional as F

import mixlab_b200
from mixlab_b200 import _lib, ops

BF16, F32 = "bf16", "f32"
DT = {BF16: torch.bfloat16, F32: torch.float32}


def listed():
    return [
        # serving, one user: the smallest call there is; 1 MB of state, so latency and launches count
        dict(name="decode_one", kind="decode", io=BF16, N=1, H=16, Dk=128, Dv=128),
        # serving, a full batch: the benchmark's decode configuration
        dict(name="decode_256", kind="decode", io=BF16, N=256, H=16, Dk=128, Dv=128),
        # the parity configuration: a short float32 forward, the reference's only data type
        dict(name="forward_f32_short", kind="scan", io=F32, mode="forward", operands=F32, log_gate=True,
             B=2, T=256, H=4, Dk=64, Dv=64),
        # the reference's own scan benchmark in its own data type, gates as multiplicative decays
        dict(name="train_f32_ref", kind="scan", io=F32, mode="train", operands=F32, log_gate=False,
             B=4, T=1024, H=4, Dk=64, Dv=128),
        # one prompt of a length that is no multiple of anything; the final state goes on to decode
        dict(name="prefill_ragged", kind="scan", io=BF16, mode="forward", operands=BF16, log_gate=True,
             B=1, T=1531, H=16, Dk=128, Dv=128),
        # the headline training configuration
        dict(name="train_bf16", kind="scan", io=BF16, mode="train", operands=BF16, log_gate=True,
             B=8, T=4096, H=16, Dk=128, Dv=128),
        # a trainer that keeps float32 tensors and accepts bf16 operands
        dict(name="train_f32_tensors", kind="scan", io=F32, mode="train", operands=BF16, log_gate=False,
             B=4, T=2048, H=16, Dk=128, Dv=128),
        # a gated_deltanet layer of the hybrid language model: 16 heads of 64 columns, sequences of 2048
        dict(name="gdn_layer_d64", kind="gdn_layer", io=BF16, B=16, T=2048, H=16, Dk=64, Dv=64),
        # the Mamba-3 training configuration
        dict(name="mamba3_train", kind="mamba3", io=BF16, mode="train", B=8, T=4096, D=2048, N=128, G=1, nheads=32),
        # the shape the reference publishes for its Mamba-3 scan, float32, per-channel parameters
        dict(name="mamba3_ref", kind="mamba3", io=F32, mode="train", B=2, T=1024, D=128, N=16, G=4, nheads=0),
        # a canonical Mamba-3 layer of the reference's larger training run, float32, per-channel parameters
        dict(name="mamba3_layer_f32", kind="mamba3_layer", io=F32, B=1, T=4096, D=448, N=16, G=4, nheads=0),
        # host tensors in, host tensors out
        dict(name="host_train", kind="host", io=BF16, B=2, T=2048, H=16, Dk=128, Dv=128),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# the largest amount of each kind: elements of state for decode, token * head * columns (or token * channel) elsewhere
_STATE_MOST = 256 * 16 * 128 * 128
_BF16_MOST = 8 * 4096 * 16
_F32_MOST = 4 * 1024 * 4


def draw(rng):
    kind = rng.choice(("decode", "scan", "scan", "scan", "gdn_layer", "mamba3", "mamba3", "mamba3_layer", "host"))
    if kind == "decode":
        c = dict(kind=kind, io=rng.choice((BF16, BF16, F32)), N=_log_int(rng, 1, 256), H=rng.choice((4, 8, 12, 16)),
                 Dk=rng.choice((64, 128, 128)), Dv=rng.choice((64, 128, 128)))
    elif kind == "scan":
        c = dict(kind=kind, io=rng.choice((BF16, BF16, F32)), mode=rng.choice(("forward", "train")))
        c["operands"] = BF16 if c["io"] == BF16 or rng.random() < 0.3 else F32
        c["log_gate"] = rng.random() < 0.5
        if c["operands"] == F32:
            c.update(H=rng.choice((1, 2, 4, 8)), Dk=8 * rng.randint(2, 16), Dv=8 * rng.randint(2, 16), B=_log_int(rng, 1, 8))
            most = _F32_MOST
        else:
            c.update(H=rng.choice((4, 8, 16)), Dk=rng.choice((64, 96, 128, 128)), Dv=rng.choice((64, 96, 128, 128)),
                     B=_log_int(rng, 1, 16))
            most = _BF16_MOST
        c["T"] = _log_int(rng, 33, min(4096, most // (c["B"] * c["H"])))
    elif kind == "gdn_layer":
        c = dict(kind=kind, io=rng.choice((BF16, BF16, F32)), B=_log_int(rng, 1, 16), H=rng.choice((4, 8, 16)))
        c["Dk"] = c["Dv"] = rng.choice((64, 64, 128))
        most = _BF16_MOST if c["io"] == BF16 else _F32_MOST
        c["T"] = _log_int(rng, 65, min(4096, most // (c["B"] * c["H"])))
    elif kind in ("mamba3", "mamba3_layer"):
        c = dict(kind=kind)
        if kind == "mamba3":
            c["mode"] = rng.choice(("forward", "train", "train"))
        if rng.random() < 0.5:  # heads of 64 channels that share their parameters, bf16
            nheads = rng.choice((8, 16, 32))
            c.update(io=BF16, B=_log_int(rng, 1, 8), D=64 * nheads, N=128, G=1, nheads=nheads)
            c["T"] = _log_int(rng, 65, min(4096, 8 * 4096 * 2048 // (c["B"] * c["D"])))
        else:                   # the reference's per-channel layout, float32
            c.update(io=F32, B=_log_int(rng, 1, 4), D=rng.choice((128, 256, 448)), N=16, G=rng.choice((1, 2, 4)), nheads=0)
            c["T"] = _log_int(rng, 65, min(4096, 4096 * 448 // (c["B"] * c["D"])))
    else:
        c = dict(kind=kind, io=BF16, B=_log_int(rng, 1, 4), H=rng.choice((8, 16)), Dk=128, Dv=128)
        c["T"] = _log_int(rng, 129, 2 * 2048 * 16 // (c["B"] * c["H"]))
    return c


# ------------------------------------------------------------------ inputs
class _Draw:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device="cuda")

    def unit(self, *shape):
        return F.normalize(self.normal(*shape), dim=-1)


def _scan_inputs(r, lead, Dk, Dv, io, log_gate, grad):
    """q, k of unit length, v normal, beta a sigmoid, the decay's logarithm a negative softplus of normals."""
    s = dict(q=r.unit(*lead, Dk).to(io), k=r.unit(*lead, Dk).to(io), v=r.normal(*lead, Dv).to(io),
             beta=torch.sigmoid(r.normal(*lead)))
    g = -F.softplus(r.normal(*lead))
    s["gate"] = g if log_gate else g.exp()
    if grad:
        s["d_out"] = r.normal(*lead, Dv).to(io)
    return s


def _mamba3_inputs(r, c, io):
    """dt before its softplus around -2, decay rates between 1 and 16, angles over the whole circle."""
    B, T, D, N, G, nh = c["B"], c["T"], c["D"], c["N"], c["G"], c["nheads"]
    s = dict(x=r.normal(B, T, D).to(io), b=r.normal(B, T, G, N).to(io), c=r.normal(B, T, G, N).to(io))
    per = (B, T, nh or D)
    s["dt"] = -2.0 + 0.5 * r.normal(*per)
    s["lam"] = r.normal(*per)
    s["theta"] = r.uniform(-math.pi, math.pi, *per) if nh else r.uniform(-math.pi, math.pi, B, T, D, N // 2)
    s["a_log"] = r.uniform(0.0, math.log(16.0), nh) if nh else r.uniform(0.0, math.log(16.0), D, N)
    return s


class _HostContext:
    """The device arena and streams a program on host buffers creates once."""

    def __init__(self, nbytes):
        self.handle = ctypes.c_void_p()
        _lib.check(mixlab_b200.lib().mxb_host_ctx_create(torch.cuda.current_device(), nbytes, ctypes.byref(self.handle)),
                   "mxb_host_ctx_create")

    def __del__(self):
        if self.handle:
            mixlab_b200.lib().mxb_host_ctx_destroy(self.handle)


def prepare(case, seed):
    c, r = case, _Draw(seed)
    io, kind = DT[c["io"]], c["kind"]
    s = dict(case=c)
    if kind == "decode":
        s.update(_scan_inputs(r, (c["N"], c["H"]), c["Dk"], c["Dv"], io, True, False))
        s["state"] = 0.02 * r.normal(c["N"], c["H"], c["Dk"], c["Dv"])
        s["out"] = torch.empty_like(s["v"])
    elif kind == "scan":
        s.update(_scan_inputs(r, (c["B"], c["T"], c["H"]), c["Dk"], c["Dv"], io, c["log_gate"], c["mode"] == "train"))
        s["flags"] = _lib.MXB_GDN_F32_IO_BF16_OPERANDS if c["io"] == F32 and c["operands"] == BF16 else 0
    elif kind == "gdn_layer":
        B, T, H, Dk, Dv = c["B"], c["T"], c["H"], c["Dk"], c["Dv"]
        s["proj"] = [r.normal(B, T, H * Dk).to(io), r.normal(B, T, H * Dk).to(io), r.normal(B, T, H * Dv).to(io),
                     0.4 * r.normal(4, H * Dk), 0.4 * r.normal(4, H * Dk), 0.4 * r.normal(4, H * Dv),
                     r.normal(B, T, H), r.normal(B, T, H), 0.5 * r.normal(H), 0.3 * r.normal(H), H, Dk, Dv]
        s["z"], s["o_norm"] = r.normal(B, T, H * Dv).to(io), 1 + 0.2 * r.normal(Dv)
        s["dy"] = r.normal(B, T, H * Dv).to(io)
    elif kind == "mamba3":
        s.update(_mamba3_inputs(r, c, io))
        if c["mode"] == "train":
            s["dy"] = r.normal(c["B"], c["T"], c["D"]).to(io)
    elif kind == "mamba3_layer":
        B, T, D, N, G = c["B"], c["T"], c["D"], c["N"], c["G"]
        s.update(_mamba3_inputs(r, c, io))
        s["b_proj"], s["c_proj"] = s.pop("b").view(B, T, G * N), s.pop("c").view(B, T, G * N)
        s.update(conv_w=0.4 * r.normal(D, 4), b_scale=1 + 0.2 * r.normal(N), c_scale=1 + 0.2 * r.normal(N),
                 b_bias=0.3 * r.normal(G * N), c_bias=0.3 * r.normal(G * N), post_norm=1 + 0.2 * r.normal(D),
                 z=r.normal(B, T, D).to(io), dout=r.normal(B, T, D).to(io))
    else:
        B, T, H, Dk, Dv = c["B"], c["T"], c["H"], c["Dk"], c["Dv"]
        d = _scan_inputs(r, (B, T, H), Dk, Dv, io, True, True)
        s["host"] = {n: t.cpu().pin_memory() for n, t in d.items()}
        s["res"] = {n: torch.empty_like(s["host"][like], pin_memory=True) for n, like in
                    (("out", "v"), ("dq", "q"), ("dk", "k"), ("dv", "v"), ("dbeta", "beta"), ("dgate", "gate"))}
        s["desc"] = mixlab_b200.GdnDesc(B, T, H, Dk, Dv, 64, mixlab_b200.MXB_BF16, 1, 0)
        need = mixlab_b200.lib().mxb_gdn_bwd_workspace_bytes(ctypes.byref(s["desc"]))
        s["ctx"] = _HostContext(need + 12 * B * T * H * max(Dk, Dv) * 2 + (64 << 20))
    return s


# ------------------------------------------------------------------ one pass
def _run_gdn_layer(s):
    # Forward, then backward.  The scan's backward recomputes its intermediates: the workspace that would hold them is
    # shared by the operators that run in between (in a model: those of the other layers).
    q, k, v, beta, gate = ops.gdn_block_pre(*s["proj"], gate_is_log=True)
    o = ops.gated_delta_scan(q, k, v, beta, gate, gate_is_log=True)
    y = ops.gdn_block_post(o, s["z"], s["o_norm"])
    gp = ops.gdn_block_post_backward(o, s["z"], s["o_norm"], s["dy"])
    gs = ops.gated_delta_scan_backward(q, k, v, beta, gate, gp["do"], gate_is_log=True)
    gi = ops.gdn_block_pre_backward(*s["proj"], gs["dq"], gs["dk"], gs["dv"], gs["dbeta"], gs["dgate"], gate_is_log=True)
    return dict(y=y, dz=gp["dz"], do_norm=gp["do_norm"], **gi)


def _run_mamba3_layer(s):
    c = s["case"]
    G, N, nh = c["G"], c["N"], c["nheads"]
    x = ops.mamba3_block_conv(s["x"], s["conv_w"])
    b, cc = ops.mamba3_block_bc(s["b_proj"], s["c_proj"], s["b_scale"], s["c_scale"], s["b_bias"], s["c_bias"], G, N)
    scan = (x, s["dt"], s["lam"], s["theta"], s["a_log"], b, cc)
    y = ops.mamba3_selective_scan(*scan, nheads=nh)
    out = ops.mamba3_block_post(y, s["z"], s["post_norm"])
    gp = ops.mamba3_block_post_backward(y, s["z"], s["post_norm"], s["dout"])
    gs = ops.mamba3_selective_scan_backward(*scan, gp["dy"], nheads=nh)
    gb = ops.mamba3_block_bc_backward(s["b_proj"], s["c_proj"], s["b_scale"], s["c_scale"], gs["db"], gs["dc"], G, N)
    gc = ops.mamba3_block_conv_backward(s["x"], s["conv_w"], gs["dx"])
    return dict(out=out, dz=gp["dz"], dpost_norm=gp["dpost_norm"], ddt=gs["ddt"], dlambda=gs["dlambda"],
                dtheta=gs["dtheta"], da_log=gs["da_log"], **gb, **gc)


def _run_host(s):
    h, r = s["host"], s["res"]
    p = [ctypes.c_void_p(t.data_ptr()) for t in (h["q"], h["k"], h["v"], h["beta"], h["gate"], r["out"], h["d_out"],
                                                 r["dq"], r["dk"], r["dv"], r["dbeta"], r["dgate"])]
    _lib.check(mixlab_b200.lib().mxb_host_gdn(s["ctx"].handle, ctypes.byref(s["desc"]), *p), "mxb_host_gdn")
    return r


def run(state):
    s = state
    c = s["case"]
    kind = c["kind"]
    if kind == "decode":
        out = ops.gated_delta_decode_step(s["state"], s["q"], s["k"], s["v"], s["beta"], s["gate"], gate_is_log=True,
                                          out=s["out"])
        return dict(out=out, state=s["state"])
    if kind == "scan":
        args, kw = (s["q"], s["k"], s["v"], s["beta"], s["gate"]), dict(gate_is_log=c["log_gate"], flags=s["flags"])
        if c["mode"] == "forward":
            out, final = ops.gated_delta_scan(*args, 64, return_final_state=True, **kw)
            return dict(out=out, final=final)
        out = ops.gated_delta_scan(*args, 64, save_for_backward=True, **kw)
        g = ops.gated_delta_scan_backward(*args, s["d_out"], 64, use_saved=True, **kw)
        return dict(out=out, **g)
    if kind == "mamba3":
        args = (s["x"], s["dt"], s["lam"], s["theta"], s["a_log"], s["b"], s["c"])
        if c["mode"] == "forward":
            return ops.mamba3_selective_scan(*args, nheads=c["nheads"])
        y = ops.mamba3_selective_scan(*args, nheads=c["nheads"], save_for_backward=True)
        g = ops.mamba3_selective_scan_backward(*args, s["dy"], nheads=c["nheads"], use_saved=True)
        return dict(y=y, **g)
    if kind == "gdn_layer":
        return _run_gdn_layer(s)
    if kind == "mamba3_layer":
        return _run_mamba3_layer(s)
    return _run_host(s)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Every input read once and every output written once; arithmetic of the plain recurrences (seven operations per
    state element and token forward, twice that backward)."""
    c = case
    kind, e = c["kind"], 2 if c["io"] == BF16 else 4
    if kind == "decode":
        per = 2 * c["Dk"] * c["Dv"] * 4 + (2 * c["Dk"] + 2 * c["Dv"]) * e + 8
        return dict(bytes=c["N"] * c["H"] * per, flops=7 * c["N"] * c["H"] * c["Dk"] * c["Dv"])
    if kind in ("scan", "gdn_layer", "host"):
        n, Dk, Dv = c["B"] * c["T"] * c["H"], c["Dk"], c["Dv"]
        if kind == "gdn_layer":  # projections, z, dy, gate inputs in; y and the gradients of all of them out
            return dict(bytes=n * (e * (4 * Dk + 5 * Dv) + 16), flops=3 * n * (7 * Dk * Dv + 30 * (2 * Dk + 2 * Dv)))
        if kind == "scan" and c["mode"] == "forward":
            return dict(bytes=n * (e * (2 * Dk + 2 * Dv) + 8) + c["B"] * c["H"] * Dk * Dv * 4, flops=7 * n * Dk * Dv)
        return dict(bytes=n * (e * (4 * Dk + 4 * Dv) + 16), flops=21 * n * Dk * Dv)
    n, D, N, GN, nh = c["B"] * c["T"], c["D"], c["N"], c["G"] * c["N"], c["nheads"]
    scalars = 4 * 3 * nh if nh else 4 * (2 * D + D * N // 2)
    flops = 7 * n * D * N
    if kind == "mamba3":
        if c["mode"] == "forward":
            return dict(bytes=n * (e * (2 * D + 2 * GN) + scalars), flops=flops)
        return dict(bytes=n * (e * (4 * D + 4 * GN) + 2 * scalars), flops=3 * flops)
    return dict(bytes=n * (e * (6 * D + 4 * GN) + 2 * scalars), flops=3 * flops + 3 * n * (40 * D + 20 * GN))


def tolerance(case):
    """Two correct implementations: float32 sums of a long recurrence in another order differ by up to 1e-4 (the bound
    the parity tests use), bf16 outputs of float32 arithmetic by roundings of single values, and bf16 tensor-core
    operands by 1e-2 in a forward and 2e-2 in gradients that pass through several rounded intermediates."""
    c = case
    if c["kind"] == "decode":
        return {"rel": 4e-3 if c["io"] == BF16 else 1e-5}
    if c["io"] == F32 and c.get("operands", F32) == F32:
        return {"rel": 1e-4}
    return {"rel": 1e-2 if c.get("mode") == "forward" else 2e-2}
