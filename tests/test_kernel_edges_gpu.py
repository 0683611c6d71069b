"""The kernels' own edges: shapes around tiles, windows, runs and the lines of the dispatch, against the CPU oracle."""
import ctypes as C

import pytest
import torch

import mixlab_b200
from mixlab_b200 import _lib, ops
from oracle import gdn, inputs
from oracle import mamba3 as oracle_mamba3
from tests import test_gdn_block_gpu as blocks
from tests import test_mamba3_gpu as mamba
from tests.util import assert_close

pytestmark = pytest.mark.gpu
F32, BF16 = torch.float32, torch.bfloat16
TOL = {F32: 1e-4, BF16: 2e-2}
GRADS = ("dq", "dk", "dv", "dbeta", "dgate", "dh0")


def _dev(t):
    return t.to("cuda").contiguous()


def _check_scan(B, T, H, K, V, io, chunk=64, offset=0):
    """Forward, backward with recompute and backward from the saved forward, with both states, at `offset` elements from
    an aligned base."""
    a = inputs.gdn_inputs(B, T, H, K, V, seed=91, io_dtype=io, with_grad_out=True, with_h0=True)
    f = {n: t.double() for n, t in a.items()}
    want = gdn.scan_grads(f["q"], f["k"], f["v"], f["beta"], f["g"], f["d_out"], f["d_state"], f["h0"], gate_is_log=True)

    def put(t):
        if not offset:
            return _dev(t)
        flat = torch.empty(t.numel() + offset, dtype=t.dtype, device="cuda")[offset:]
        return flat.copy_(t.reshape(-1)).view(t.shape)

    args = tuple(put(a[n]) for n in ("q", "k", "v", "beta", "g"))
    d_out, h0, d_state = put(a["d_out"]), _dev(a["h0"]), _dev(a["d_state"])
    kw = dict(gate_is_log=True, h0=h0)
    ref = ops.gated_delta_scan_backward(*args, d_out, chunk, d_final_state=d_state, **kw)
    ref = {n: ref[n].clone() for n in GRADS}
    o, s = ops.gated_delta_scan(*args, chunk, return_final_state=True, **kw)
    saved = ops.gated_delta_scan(*args, chunk, save_for_backward=True, **kw)
    got = ops.gated_delta_scan_backward(*args, d_out, chunk, d_final_state=d_state, use_saved=True, **kw)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert torch.equal(o, saved)
    assert_close(o, want["out"], TOL[io], "out")
    assert_close(s, want["state"], TOL[io], "final_state")
    for n in GRADS:
        assert torch.equal(got[n], ref[n]), n
        assert_close(got[n], want[n], TOL[io], n)


@pytest.mark.parametrize("shape,chunk,offset", [
    ((1, 65, 1, 16, 24), 64, 0),       # narrowest column slabs, ragged in columns and steps
    ((2, 64, 2, 128, 128), 64, 0),     # two K tiles, whole chunks
    ((3, 63, 4, 96, 40), 64, 0),       # middle slab width, K between the tiles
    ((8, 66, 8, 64, 64), 64, 0),       # enough heads for the widest slabs
    ((1, 70, 2, 18, 20), 64, 0),       # rows that no tensor copy can move
    ((1, 70, 2, 16, 24), 64, 1),       # nor from such a base
    ((2, 70, 2, 32, 16), 16, 0), ((1, 1, 1, 8, 8), 64, 0),
])
def test_float32_scan(shape, chunk, offset):
    _check_scan(*shape, F32, chunk, offset)


@pytest.mark.parametrize("T,chunk", [(64, 64), (50, 64), (33, 33), (16, 16), (1, 64)])
def test_float32_decay_matrix(T, chunk):
    """Unit vectors for keys, their sum for every query, unit vectors for values, beta 1: the output of a chunk is
    exp(G_i - G_j), G the float32 sums of the log gates taken one after the other (sums in another order are 1e-5 away).
    What is left is expf: 2 ulp, and an ulp for the additions of zeros."""
    B, H = 2, 8
    eye = torch.eye(T, 64).expand(B, H, T, 64).transpose(1, 2)
    q = torch.ones(B, T, H, 64)
    gate = -torch.nn.functional.softplus(torch.randn(B, T, H, generator=torch.Generator().manual_seed(95)))
    out = ops.gated_delta_scan(_dev(q), _dev(eye), _dev(eye), _dev(torch.ones(B, T, H)), _dev(gate), chunk, gate_is_log=True)
    sums, acc = [], torch.zeros(B, H)
    for t in range(T):
        acc = acc + gate[:, t]
        sums.append(acc)
    G = torch.stack(sums, 1)                                     # [B,T,H]
    diff = G[:, :, None] - G[:, None]                            # float32, [B,T,T,H]
    assert float(diff.min()) > -80
    want = torch.exp(diff.double()) * torch.tril(torch.ones(T, T))[None, :, :, None].double()
    got = out.double().cpu()[..., :T].permute(0, 1, 3, 2)
    assert float((got - want).abs().div(want.clamp_min(1e-30)).max()) <= 3 * 2 ** -23


@pytest.mark.parametrize("log_gate", [True, False])
@pytest.mark.parametrize("shape", [(2, 256, 4, 64, 64), (1, 300, 2, 128, 256), (2, 513, 3, 96, 200), (2, 70, 2, 16, 24)])
def test_float32_scan_loses_no_more_than_plain_float32(shape, log_gate):
    """Every result is as close to the float64 oracle as the same formulas in plain float32 are (a quarter more for sums in
    another order)."""
    a = inputs.gdn_inputs(*shape, seed=5, io_dtype=F32, with_grad_out=True, with_h0=True)
    gate = a["g"] if log_gate else torch.exp(a["g"])

    def oracle(dtype):
        f = {n: t.to(dtype) for n, t in a.items()}
        return gdn.scan_grads(f["q"], f["k"], f["v"], f["beta"], gate.to(dtype), f["d_out"], f["d_state"], f["h0"],
                              gate_is_log=log_gate, chunk_size=64)

    want, plain = oracle(torch.float64), oracle(F32)
    args, kw = tuple(_dev(t) for t in (a["q"], a["k"], a["v"], a["beta"], gate)), dict(gate_is_log=log_gate, h0=_dev(a["h0"]))
    got = ops.gated_delta_scan_backward(*args, _dev(a["d_out"]), 64, d_final_state=_dev(a["d_state"]), **kw)
    got["out"], got["state"] = ops.gated_delta_scan(*args, 64, return_final_state=True, **kw)
    off = lambda x, w: float((x.double().cpu() - w).norm() / w.norm())
    for n in GRADS + ("out", "state"):
        assert off(got[n], want[n]) <= 1.25 * off(plain[n], want[n]), n


@pytest.mark.parametrize("shape", [
    (1, 1, 1, 128, 128), (1, 64, 2, 128, 96), (2, 129, 3, 96, 72), (1, 193, 2, 64, 128),   # split columns
    (2, 65, 37, 128, 128),             # the most heads that split
    (3, 65, 25, 128, 128),             # the fewest that do not
    (1, 1, 1, 64, 64), (2, 63, 3, 64, 64), (1, 64, 2, 64, 64), (1, 130, 5, 64, 64),        # 64-wide kernels
])
def test_tensor_core_scan(shape):
    _check_scan(*shape, BF16)


@pytest.mark.parametrize("dims", [(1, 1, 4, 4), (2, 3, 256, 8), (1, 2, 64, 36), (2, 2, 100, 28), (1, 1, 128, 256),
                                  (70, 5, 64, 96)])
@pytest.mark.parametrize("io", [F32, BF16])
def test_decode_slabs(dims, io):
    N, H, K, V = dims
    a = inputs.gdn_decode_inputs(N, H, K, V, 1, seed=92, io_dtype=io)
    x = {n: a[n][0] for n in ("q", "k", "v", "beta", "g")}
    o_ref, st_ref = gdn.decode_step(a["state"].double(), x["q"].double(), x["k"].double(), x["v"].double(),
                                    x["beta"].double(), torch.exp(x["g"].double()))
    st = _dev(a["state"].clone())
    o = ops.gated_delta_decode_step(st, *(_dev(x[n]) for n in ("q", "k", "v", "beta", "g")), gate_is_log=True)
    assert_close(o, o_ref, TOL[io], "out")
    assert_close(st, st_ref, TOL[F32], "state")


@pytest.mark.parametrize("cfg", [(1, 31, 1, 64, 64), (1, 33, 5, 8, 64), (2, 129, 2, 64, 8), (1, 65, 3, 32, 48)])
@pytest.mark.parametrize("io", [F32, BF16])
def test_block_stages(cfg, io):
    """Runs of steps that end inside a sequence, rows narrower than a warp, queries and values of different widths."""
    blocks.test_block_pre_forward_and_gradients(cfg, io, True)
    B, T, H, _, V = cfg
    blocks.test_block_post_forward_and_gradients((B, T, H, V), io)


@pytest.mark.parametrize("B,T,H,K,V", [(21846, 2, 1, 8, 8), (65535, 1, 1, 8, 16), (70000, 1, 1, 8, 8), (1, 65535 * 128 + 1, 1, 8, 8)])
def test_block_stages_beyond_a_grid_axis(B, T, H, K, V):
    """More sequences than a grid axis holds for three streams, and a sequence of more tiles: the same bits as those
    sequences (or that piece of the sequence) alone; the gradients of the weights against sums over the pieces."""
    g = torch.Generator(device="cuda").manual_seed(96)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    seq = [rn(B, T, H * K).to(BF16), rn(B, T, H * K).to(BF16), rn(B, T, H * V).to(BF16)]
    conv, gates, head = [0.4 * rn(4, H * K), 0.4 * rn(4, H * K), 0.4 * rn(4, H * V)], [rn(B, T, H), rn(B, T, H)], [rn(H), rn(H)]
    grads = [rn(B, T, H, K).to(BF16), rn(B, T, H, K).to(BF16), rn(B, T, H, V).to(BF16), rn(B, T, H), rn(B, T, H)]
    args = lambda cut: [cut(t) for t in seq] + conv + [cut(t) for t in gates] + head + [H, K, V]
    whole = ops.gdn_block_pre(*args(lambda t: t), gate_is_log=True)
    back = ops.gdn_block_pre_backward(*args(lambda t: t), *grads, gate_is_log=True)
    if B > 1:
        pieces = [lambda t: t[:100].contiguous(), lambda t: t[B - 100:].contiguous(), lambda t: t[B // 2:B // 2 + 100].contiguous()]
        mid = slice(None)
    else:  # the first steps of a piece lack the steps before it, the last ones the gradients behind it
        pieces = [lambda t: t[:, T - 200:].contiguous(), lambda t: t[:, T // 2:T // 2 + 200].contiguous()]
        mid = slice(3, -3)
    for cut in pieces:
        part = ops.gdn_block_pre(*args(cut), gate_is_log=True)
        for x, y in zip(whole, part):
            assert torch.equal(cut(x)[:, mid], y[:, mid])
        pb = ops.gdn_block_pre_backward(*args(cut), *(cut(t) for t in grads), gate_is_log=True)
        for n in ("dq_proj", "dk_proj", "dv_proj", "da_raw", "db_raw"):
            assert torch.equal(cut(back[n])[:, mid], pb[n][:, mid]), n
    assert all(bool(torch.isfinite(back[n]).all()) for n in ("dconv_q", "dconv_k", "dconv_v"))
    if B > 1:  # halves of the batch add up
        halves = [ops.gdn_block_pre_backward(*args(c), *(c(t) for t in grads), gate_is_log=True)
                  for c in (lambda t: t[:B // 2].contiguous(), lambda t: t[B // 2:].contiguous())]
        for n in ("dconv_q", "dconv_k", "dconv_v", "da_log", "ddt_bias"):
            assert_close(back[n], halves[0][n].double() + halves[1][n].double(), 1e-4, n)


@pytest.mark.parametrize("shape", [(1, 2, 4, 8, 1), (1, 7, 4, 16, 1), (2, 8, 8, 16, 2), (1, 9, 4, 32, 1),
                                   (1, 24, 4, 64, 1), (1, 17, 2, 256, 1), (1, 15, 4, 6, 1), (1, 41, 3, 128, 1)])
def test_mamba3_windows(shape):
    """Windows of eight steps: none full, exactly full, one step over; vector and scalar rows, each lane count."""
    mamba.test_window_parallel_matches_serial_walk(shape)
    B, T, D, N, G = shape
    a = inputs.mamba3_inputs(B, T, D, 1, N, G=G, seed=93, per_head=False)
    dev, dy = [_dev(a[n]) for n in mamba.ARGS], _dev(a["dy"])
    kw = dict(flags=_lib.MXB_MAMBA3_WINDOW_PARALLEL)
    want = {n: t.clone() for n, t in ops.mamba3_selective_scan_backward(*dev, dy, **kw).items()}
    ops.mamba3_selective_scan(*dev, save_for_backward=True, **kw)
    got = ops.mamba3_selective_scan_backward(*dev, dy, use_saved=True, **kw)
    for n in mamba.GRADS:
        assert torch.equal(got[n], want[n]), n


def test_mamba3_windows_beyond_a_grid_axis():
    """More windows than a grid axis holds, against the serial walk.  Angles turn in the last thousand steps only: over half a
    million the two forms would round them apart.  da_log adds 5e5 terms, in the serial walk one after the other in
    float32 (a random walk of 4e-5, more where they lean one way): 1e-3."""
    B, T, D, N, G = 1, 65535 * 8 + 9, 4, 4, 1
    a = inputs.mamba3_inputs(B, T, D, 1, N, G=G, seed=97, per_head=False)
    a["theta"][:, :T - 1000] = 0
    dev, dy = [_dev(a[n]) for n in mamba.ARGS], _dev(a["dy"])
    serial, default = dict(flags=_lib.MXB_MAMBA3_SERIAL_WALK), {}
    n0 = mixlab_b200.lib().mxb_launch_count()
    y = ops.mamba3_selective_scan(*dev, **default)
    assert mixlab_b200.lib().mxb_launch_count() - n0 > 1      # the windows, not the walk of one launch
    assert_close(y, ops.mamba3_selective_scan(*dev, **serial).double(), 1e-5, "y")
    got, want = (ops.mamba3_selective_scan_backward(*dev, dy, **kw) for kw in (default, serial))
    for n in mamba.GRADS:
        assert_close(got[n], want[n].double(), 1e-3 if n == "da_log" else 1e-4, n)


@pytest.mark.parametrize("cfg", [(1, 63, 1, 1), (2, 65, 3, 3), (1, 129, 2, 2)])
def test_mamba3_chunks(cfg):
    """Chunks of 64 steps, one short, one over; one head per group."""
    mamba.test_chunked_tensor_core_kernels(cfg)


def test_mamba3_chunks_beyond_a_grid_axis():
    """More chunks than the 65,535 blocks of a grid's y axis, against the recurrent kernels on the last 2048 steps alone: over
    the last thousand the states before that piece have decayed (exp(-80) and less), and only differences of angles count."""
    T, P, N, piece, tail = 65535 * 64 + 65, 64, 128, 2048, 1000
    g = torch.Generator(device="cuda").manual_seed(98)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    # (the pieces of a sequence this long that matter are its last steps: 64 k random steps, repeated)
    wide = lambda w: rn(1, 1 << 16, w).to(BF16).repeat(1, T // (1 << 16) + 1, 1)[:, :T].contiguous()
    x, dy, b, c = wide(P), wide(P), wide(N).view(1, T, 1, N), wide(N).view(1, T, 1, N)
    dt, lam, theta, a_log = rn(1, T, 1) * 0.5 - 2, rn(1, T, 1), rn(1, T, 1), torch.zeros(1, device="cuda")
    y = ops.mamba3_selective_scan(x, dt, lam, theta, a_log, b, c, nheads=1, save_for_backward=True)
    got = ops.mamba3_selective_scan_backward(x, dt, lam, theta, a_log, b, c, dy, nheads=1, use_saved=True)
    assert ops.device_status() == 0
    end = lambda t: t[:, T - piece:].contiguous()
    part = (end(x), end(dt), end(lam), end(theta), a_log, end(b), end(c))
    kw = dict(nheads=1, flags=_lib.MXB_MAMBA3_RECURRENT_KERNELS)
    y_r = ops.mamba3_selective_scan(*part, **kw)
    want = ops.mamba3_selective_scan_backward(*part, end(dy), **kw)
    assert_close(y[:, -tail:], y_r[:, -tail:].double(), 2e-2, "y")
    for n in mamba.GRADS:
        if n != "da_log":  # (a sum over all steps)
            assert_close(got[n][:, -tail:], want[n][:, -tail:].double(), 2e-2, n)
    assert bool(torch.isfinite(got["da_log"]).all())


@pytest.mark.parametrize("B,T,H,arena_mb", [(1, 130, 4, 256), (4, 600, 8, 256), (4, 600, 8, 40), (2, 2100, 8, 256)])
def test_host_slicing(B, T, H, arena_mb):
    """Slices of whole sequences and of groups of heads, two to four in flight, and finer ones where the arena is small:
    the results of the device entry points, bit for bit."""
    lib = mixlab_b200.lib()
    a = inputs.gdn_inputs(B, T, H, 128, 128, seed=94, io_dtype=BF16, with_grad_out=True)
    names = ("q", "k", "v", "beta", "g")
    dev = [_dev(a[n]) for n in names]
    want = dict(out=ops.gated_delta_scan(*dev, 64, gate_is_log=True).clone())
    want.update(ops.gated_delta_scan_backward(*dev, _dev(a["d_out"]), 64, gate_is_log=True))
    host = {n: a[n].contiguous().pin_memory() for n in names + ("d_out",)}
    res = {n: torch.empty_like(host[m]).pin_memory() for n, m in
           (("out", "v"), ("dq", "q"), ("dk", "k"), ("dv", "v"), ("dbeta", "beta"), ("dgate", "g"))}
    p = lambda t: C.c_void_p(t.data_ptr())
    ctx = C.c_void_p()
    assert lib.mxb_host_ctx_create(0, arena_mb << 20, C.byref(ctx)) == 0
    try:
        d = mixlab_b200.GdnDesc(B, T, H, 128, 128, 64, mixlab_b200.MXB_BF16, 1, 0)
        assert lib.mxb_host_gdn(ctx, C.byref(d), *(p(host[n]) for n in names), p(res["out"]), p(host["d_out"]),
                                *(p(res[n]) for n in ("dq", "dk", "dv", "dbeta", "dgate"))) == 0
    finally:
        lib.mxb_host_ctx_destroy(ctx)
    for n, t in res.items():
        assert torch.equal(t, want[n].cpu()), n


@pytest.mark.parametrize("T,K,V,batches", [
    (150, 128, 128, (2, 8, 18)),   # of 4 heads: 16 and 32 columns of the state per CTA, the tcgen05 pass of 64 columns
    (64, 128, 72, (3, 9)),         # one whole chunk, columns past the values' width
    (449, 72, 128, (1, 9)),        # more chunks than buffers, rows past the keys' width
    (130, 64, 64, (9, 18)),        # heads of 64 columns: 16 and 32 columns per CTA
])
def test_gdn_state_passes_agree_bit_for_bit(T, K, V, batches):
    """Sequences of a batch that fills the GPU (tcgen05 state passes) and the first few of them alone (mma.sync passes of
    16 and 32 columns): the same roundings and the same order of sums, so the same bits.  The oracle pins either route."""
    a = inputs.gdn_inputs(40, T, 4, K, V, seed=17, io_dtype=BF16, with_grad_out=True, with_h0=True)
    d = {n: _dev(t) for n, t in a.items()}

    def run(nb):
        x = {n: t[:nb] for n, t in d.items()}
        args = tuple(x[n] for n in ("q", "k", "v", "beta", "g"))
        kw = dict(gate_is_log=True, h0=x["h0"])
        o, s = ops.gated_delta_scan(*args, 64, return_final_state=True, **kw)
        saved = ops.gated_delta_scan(*args, 64, save_for_backward=True, **kw)
        g = ops.gated_delta_scan_backward(*args, x["d_out"], 64, d_final_state=x["d_state"], use_saved=True, **kw)
        torch.cuda.synchronize()
        assert ops.device_status() == 0 and torch.equal(o, saved)
        return dict(out=o, state=s, **g)

    whole = run(40)
    for nb in batches:
        part = run(nb)
        for n in whole:
            assert torch.equal(whole[n][:nb], part[n]), (nb, n)


@pytest.mark.parametrize("B,T,K,V", [
    (2, 150, 128, 128), (9, 65, 128, 72), (18, 130, 72, 128), (40, 70, 128, 128),   # state passes of 16, 32, 64, 128 columns
    (2, 100, 64, 64), (18, 64, 64, 64), (40, 66, 64, 64), (40, 66, 96, 88),         # heads of 64 columns; widths between
])
def test_float32_results_of_the_tensor_core_kernels(B, T, K, V):
    """Float32 tensors through the tensor-core kernels: every state pass and chunk kernel writes its rounded results as
    float32 itself, so they are the bf16 entry's results, widened (gradients from a saved and from a recomputed forward)."""
    a = inputs.gdn_inputs(B, T, 4, K, V, seed=23, io_dtype=BF16, with_grad_out=True)
    low = [_dev(a[n]) for n in ("q", "k", "v", "beta", "g")]
    wide = [t.float() for t in low]
    d_low = _dev(a["d_out"])
    kw, flag = dict(gate_is_log=True), _lib.MXB_GDN_F32_IO_BF16_OPERANDS
    want_o = ops.gated_delta_scan(*low, 64, **kw)
    want = ops.gated_delta_scan_backward(*low, d_low, 64, **kw)
    o = ops.gated_delta_scan(*wide, 64, flags=flag, save_for_backward=True, **kw)
    saved = ops.gated_delta_scan_backward(*wide, d_low.float(), 64, flags=flag, use_saved=True, **kw)
    again = ops.gated_delta_scan_backward(*wide, d_low.float(), 64, flags=flag, **kw)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert o.dtype == F32 and torch.equal(o, want_o.float())
    for n in ("dq", "dk", "dv", "dbeta", "dgate"):
        assert torch.equal(saved[n], want[n].float()), n
        assert torch.equal(again[n], want[n].float()), n


@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cfg", [(1, 4801, 448), (2, 9, 512), (1, 7, 520), (1, 1, 8)])
def test_block_post_rows_on_both_sides_of_a_warp(cfg, io):
    """Rows of up to 512 channels belong to a warp, wider ones to a CTA; more partial rows than one round of the column sums."""
    from test_mamba3_block_gpu import test_post_forward_and_gradients
    test_post_forward_and_gradients(cfg, io)


@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cfg", [(1, 65, 2, 8), (2, 129, 3, 24), (1, 33, 1, 32), (1, 70, 2, 40), (3, 1700, 1, 16), (1, 17, 4, 104)])
def test_block_bc_rows_of_every_lane_group(cfg, io):
    """2, 4, 8 and 16 lanes a row, whole and partly filled, with ragged numbers of rows."""
    from test_mamba3_block_gpu import test_bc_norm_forward_and_gradients
    test_bc_norm_forward_and_gradients(cfg, io)


@pytest.mark.parametrize("T", [1, 64, 65, 130, 257])
@pytest.mark.parametrize("G", [1, 2])
def test_mamba3_states_and_output_in_one_kernel(T, G):
    """More (batch, head) pairs than SMs take one kernel for states and output, fewer take two: the same bits, and the states it
    keeps serve the backward as the recomputed ones do."""
    B, nheads = 5, 32
    a = inputs.mamba3_inputs(B, T, nheads, 64, 128, G=G, seed=61, io_dtype=BF16, per_head=True)
    names = ("x", "dt_raw", "lambda_raw", "theta", "a_log", "b", "c")
    args = [_dev(a[n]) for n in names]
    y = ops.mamba3_selective_scan(*args, nheads=nheads, save_for_backward=True)
    dy = _dev(a["dy"])
    saved = ops.mamba3_selective_scan_backward(*args, dy, nheads=nheads, use_saved=True)
    again = ops.mamba3_selective_scan_backward(*args, dy, nheads=nheads)
    for n in saved:
        assert torch.equal(saved[n], again[n]), n
    assert torch.equal(y, ops.mamba3_selective_scan(*args, nheads=nheads))
    for b in (0, B - 1):
        row = [t if n == "a_log" else t[b:b + 1].contiguous() for n, t in zip(names, args)]
        assert torch.equal(y[b:b + 1], ops.mamba3_selective_scan(*row, nheads=nheads))


@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 16, 63, 64, 67, 130])
def test_block_conv_long_runs(T, io):
    """Enough sequences that a lane takes 64 steps: runs that end inside, at and just behind the sequence; weights that can be read
    four taps at a time and ones that cannot (three taps, or a base that is not 16-byte aligned)."""
    from oracle import mamba3_block
    B, D = 444, 8
    g = torch.Generator().manual_seed(T)
    x, dy = torch.randn(B, T, D, generator=g).to(io), torch.randn(B, T, D, generator=g).to(io)
    flat = 0.4 * torch.randn(4 * D + 1, generator=g)
    for K, first in ((4, 0), (4, 1), (3, 0)):
        w = flat[first:first + K * D].view(D, K)
        x64, w64 = x.double().requires_grad_(True), w.double().requires_grad_(True)
        y = mamba3_block.depthwise_conv(x64, w64)
        gx, gw = torch.autograd.grad((y * dy.double()).sum(), [x64, w64])
        dw = flat.to("cuda")[first:first + K * D].view(D, K)
        assert_close(ops.mamba3_block_conv(_dev(x), dw), y.detach(), TOL[io], f"y {K} {first}")
        got = ops.mamba3_block_conv_backward(_dev(x), dw, _dev(dy))
        assert_close(got["dx"], gx, TOL[io], f"dx {K} {first}")
        assert_close(got["dw"], gw, TOL[io], f"dw {K} {first}")


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("T,step", [(40, 3), (200, 77), (1300, 900)])
def test_mamba3_windows_pass_on_angles_that_are_not_finite(T, step, bad):
    """An angle that is not finite makes the same results NaN as in the serial walk: every later angle of its pair is NaN, in its own
    window and in all that follow (one, some and all segments of the scan)."""
    a = inputs.mamba3_inputs(1, T, 16, 1, 8, G=2, seed=71, per_head=False)
    a["theta"][0, step, 5, 2] = bad
    args = [_dev(a[n]) for n in ("x", "dt_raw", "lambda_raw", "theta", "a_log", "b", "c")]
    got, want = ({"y": ops.mamba3_selective_scan(*args, flags=f), **ops.mamba3_selective_scan_backward(*args, _dev(a["dy"]), flags=f)}
                 for f in (_lib.MXB_MAMBA3_WINDOW_PARALLEL, _lib.MXB_MAMBA3_SERIAL_WALK))
    assert bool(torch.isnan(want["dx"][0, step:, 5]).all()) and not bool(torch.isnan(want["dx"][0, :, 4]).any())
    for n in want:
        assert torch.equal(torch.isnan(got[n]), torch.isnan(want[n])), n


def test_mamba3_window_angles_around_odd_multiples_of_pi():
    """The angle at a window start, read off as the sine by which the row of c has turned against the state (no decay, one input).
    Bound: the sum back in float32 2.4e-7 (as a float, and its product with 2 pi / 2^32) and that constant 1e-7, the wrap of the first
    step 2.4e-7, the sine 1.2e-7: 7e-7."""
    pi = torch.tensor([k * torch.pi for k in range(1, 256, 2)], dtype=torch.float64).float()
    above, below = torch.nextafter(pi, pi + 1), torch.nextafter(pi, pi - 1)
    X = torch.cat([pi, above, below, torch.nextafter(above, above + 1)])
    X = torch.cat([X, -X])
    D, T = X.numel(), 9
    x, theta = torch.zeros(1, T, D), torch.zeros(1, T, D, 1)
    x[:, 0], theta[0, 1, :, 0] = 1, X / 32
    dt, lam, a_log = torch.full((1, T, D), 32.0), torch.full((1, T, D), 60.0), torch.full((D, 2), -float("inf"))
    b, c = torch.tensor([1.0, 0.0]).expand(1, T, 1, 2), torch.tensor([0.0, 1.0]).expand(1, T, 1, 2)
    y = ops.mamba3_selective_scan(*map(_dev, (x, dt, lam, theta, a_log, b, c)), flags=_lib.MXB_MAMBA3_WINDOW_PARALLEL)
    err = float((y[0, 8].cpu().double() / 32 - torch.sin(X.double())).abs().max())
    assert err <= 7e-7, err


def test_mamba3_window_decays_are_as_exact_as_expf():
    """The decay of one step, read off as the state of a step that adds nothing (A = -1, so that dt is the exponent without rounding).
    Bound: two units in the last place of float32, 2.4e-7."""
    D = 1 << 14
    x, theta, lam = torch.zeros(1, 2, D), torch.zeros(1, 2, D, 1), torch.full((1, 2, D), 60.0)
    x[:, 0] = 1
    dt = torch.full((1, 2, D), 32.0)          # softplus(dt) = dt above 20
    dt[0, 1] = torch.linspace(20.5, 87, D)
    b = torch.tensor([1.0, 0.0]).expand(1, 2, 1, 2)
    y = ops.mamba3_selective_scan(*map(_dev, (x, dt, lam, theta, torch.zeros(D, 2), b, b)), flags=_lib.MXB_MAMBA3_WINDOW_PARALLEL)
    want = 32 * torch.exp(-dt[0, 1].double())
    err = float(((y[0, 1].cpu().double() - want) / want).abs().max())
    assert err <= 2.4e-7, err


def _check_windows(B, T, D, N, G, io):
    a = inputs.mamba3_inputs(B, T, D, 1, N, G=G, seed=73, io_dtype=io, per_head=False)
    names = ("x", "dt_raw", "lambda_raw", "theta", "a_log", "b", "c")
    args, kw = [_dev(a[n]) for n in names], dict(flags=_lib.MXB_MAMBA3_WINDOW_PARALLEL)
    y_ref, want = oracle_mamba3.scan_vjp(*(a[n].double() for n in names), a["dy"].double())
    assert_close(ops.mamba3_selective_scan(*args, **kw), y_ref, TOL[io], "y")
    got = ops.mamba3_selective_scan_backward(*args, _dev(a["dy"]), **kw)
    for n in want:
        assert_close(got[n], want[n], TOL[io], n)


@pytest.mark.parametrize("T", [1025, 1100, 2048])
def test_mamba3_windows_eight_to_a_segment(T):
    """Forward and reverse scans whose segments hold eight windows, the last segment whole, partly filled and the last of all."""
    _check_windows(1, T, 16, 8, 2, F32)


@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N", [16, 14])
def test_mamba3_windows_of_seven_warps(N, io):
    """Groups of 112 channels make CTAs of seven warps, and 304 of them a gradient walk that fits the GPU at once with the fewer
    registers; states that can be read two pairs at a time and ones that cannot."""
    _check_windows(1, 300, 448, N, 4, io)


@pytest.mark.parametrize("io", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T,D", [(444, 67, 136), (444, 64, 136), (444, 130, 136), (444, 67, 72), (444, 16, 128), (740, 64, 32), (741, 64, 64), (444, 67, 64),
                                   (1480, 33, 8), (16, 300, 24)])
def test_block_conv_runs_of_narrow_rows(B, T, D, io):
    """bf16 rows of up to sixteen lanes and the first wider ones, with 16, 32 and 64 steps a lane."""
    from oracle import mamba3_block
    g = torch.Generator().manual_seed(D)
    x, dy, w = torch.randn(B, T, D, generator=g).to(io), torch.randn(B, T, D, generator=g).to(io), 0.4 * torch.randn(D, 4, generator=g)
    x64, w64 = x.double().requires_grad_(True), w.double().requires_grad_(True)
    y = mamba3_block.depthwise_conv(x64, w64)
    gx, gw = torch.autograd.grad((y * dy.double()).sum(), [x64, w64])
    assert_close(ops.mamba3_block_conv(_dev(x), _dev(w)), y.detach(), TOL[io], "y")
    got = ops.mamba3_block_conv_backward(_dev(x), _dev(w), _dev(dy))
    assert_close(got["dx"], gx, TOL[io], "dx")
    assert_close(got["dw"], gw, TOL[io], "dw")


@pytest.mark.parametrize("B,NH,one", [(4, 37, False), (149, 1, True), (5, 32, True), (10, 30, True)])
def test_mamba3_states_and_output_kernels_by_pairs(B, NH, one):
    """Up to 148 (batch, head) pairs take a kernel for the states and one for the output, more take one for both (also in a second
    round of CTAs, from 297 on); a single sequence of the same inputs gives the same bits through the two."""
    a = inputs.mamba3_inputs(B, 130, NH, 64, 128, G=1, seed=62, io_dtype=BF16, per_head=True)
    names = ("x", "dt_raw", "lambda_raw", "theta", "a_log", "b", "c")
    args = [_dev(a[n]) for n in names]

    def run(args):
        n0 = mixlab_b200.lib().mxb_launch_count()
        y = ops.mamba3_selective_scan(*args, nheads=NH)
        return y, mixlab_b200.lib().mxb_launch_count() - n0

    row = [t if n == "a_log" else t[B - 1:].contiguous() for n, t in zip(names, args)]
    (y, launches), (y_row, launches_row) = run(args), run(row)
    assert launches_row - launches == (1 if one else 0)
    assert torch.equal(y[B - 1:], y_row)
