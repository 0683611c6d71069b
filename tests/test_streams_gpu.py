"""Calls on several streams, from several threads and in graphs: the cached scratch of one is not touched by another."""
import threading

import pytest
import torch

from mixlab_b200 import _lib, ops
from oracle import inputs

pytestmark = pytest.mark.gpu


def _scan_case(seed, T):
    a = inputs.gdn_inputs(2, T, 4, 128, 128, seed=seed, io_dtype=torch.bfloat16, with_grad_out=True)
    return tuple(a[n].cuda().contiguous() for n in ("q", "k", "v", "beta", "g")), a["d_out"].cuda().contiguous()


def _train(args, d_out):
    out = ops.gated_delta_scan(*args, 64, gate_is_log=True, save_for_backward=True)
    g = ops.gated_delta_scan_backward(*args, d_out, 64, gate_is_log=True, use_saved=True)
    return [out] + [g[n] for n in ("dq", "dk", "dv", "dbeta", "dgate")]


def test_saved_forwards_of_two_streams_side_by_side():
    """Two streams, each with a saved forward, then each with its backward: neither overwrites what the other saved."""
    cases = [_scan_case(s, 900) for s in (1, 2)]
    want = [[t.clone() for t in _train(*c)] for c in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    for _ in range(20):
        outs, grads = [], []
        for st, (args, _) in zip(streams, cases):
            with torch.cuda.stream(st):
                outs.append(ops.gated_delta_scan(*args, 64, gate_is_log=True, save_for_backward=True))
        for st, (args, d_out) in zip(streams, cases):
            with torch.cuda.stream(st):
                grads.append(ops.gated_delta_scan_backward(*args, d_out, 64, gate_is_log=True, use_saved=True))
        torch.cuda.synchronize()
        for o, g, w in zip(outs, grads, want):
            for x, y in zip([o] + [g[n] for n in ("dq", "dk", "dv", "dbeta", "dgate")], w):
                assert torch.equal(x, y)
    for st in streams:
        with torch.cuda.stream(st):
            assert ops.device_status() == 0


@pytest.mark.parametrize("own_stream", [True, False])
def test_threads(own_stream):
    """Threads with a stream each, and threads that share one: results of every call as if it ran alone.  On a shared
    stream another thread's call may come between a saving forward and its backward; that backward is refused."""
    cases = [_scan_case(s, 300 + 64 * s) for s in range(4)]
    want = [[t.clone() for t in _train(*c)] for c in cases]
    torch.cuda.synchronize()
    failures = []

    def work(i):
        args, d_out = cases[i]
        try:
            with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
                for _ in range(60):
                    out = ops.gated_delta_scan(*args, 64, gate_is_log=True, save_for_backward=True)
                    try:
                        g = ops.gated_delta_scan_backward(*args, d_out, 64, gate_is_log=True, use_saved=True)
                    except RuntimeError:
                        assert not own_stream
                        g = ops.gated_delta_scan_backward(*args, d_out, 64, gate_is_log=True)
                    torch.cuda.current_stream().synchronize()
                    for x, y in zip([out] + [g[n] for n in ("dq", "dk", "dv", "dbeta", "dgate")], want[i]):
                        assert torch.equal(x, y)
        except BaseException as e:  # reported by the main thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_streams_beyond_the_kept_ones():
    """More streams than keep a buffer: the one given back is the longest unused, and its saved forward is refused."""
    args, d_out = _scan_case(5, 200)
    want = [t.clone() for t in _train(args, d_out)]
    streams = [torch.cuda.Stream() for _ in range(12)]
    torch.cuda.synchronize()
    for st in streams:
        with torch.cuda.stream(st):
            ops.gated_delta_scan(*args, 64, gate_is_log=True, save_for_backward=True)
    with torch.cuda.stream(streams[0]), pytest.raises(RuntimeError):
        ops.gated_delta_scan_backward(*args, d_out, 64, gate_is_log=True, use_saved=True)
    with torch.cuda.stream(streams[-1]):
        g = ops.gated_delta_scan_backward(*args, d_out, 64, gate_is_log=True, use_saved=True)
    torch.cuda.synchronize()
    for n, w in zip(("dq", "dk", "dv", "dbeta", "dgate"), want[1:]):
        assert torch.equal(g[n], w), n


@pytest.mark.parametrize("flags,nheads", [(_lib.MXB_MAMBA3_SERIAL_WALK, 0), (_lib.MXB_MAMBA3_WINDOW_PARALLEL, 0),
                                          (_lib.MXB_MAMBA3_RECURRENT_KERNELS, 2), (0, 2)])
def test_saved_mamba3_forward_on_a_new_stream(flags, nheads):
    """A stream whose buffer nobody has used: the backward of a saving forward finds room, also where that kernel family
    saves nothing and recomputes."""
    a = inputs.mamba3_inputs(1, 130, 2, 64, 128, G=1, seed=24, io_dtype=torch.bfloat16, per_head=nheads > 0)
    args = [a[n].cuda().contiguous() for n in ("x", "dt_raw", "lambda_raw", "theta", "a_log", "b", "c")]
    dy, kw = a["dy"].cuda().contiguous(), dict(flags=flags, nheads=nheads)
    want = {n: t.clone() for n, t in ops.mamba3_selective_scan_backward(*args, dy, **kw).items()}
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream(priority=-1)):
        ops.mamba3_selective_scan(*args, save_for_backward=True, **kw)
        got = ops.mamba3_selective_scan_backward(*args, dy, use_saved=True, **kw)
    torch.cuda.synchronize()
    for n, t in want.items():
        assert torch.equal(got[n], t), n


def _capture(stream, args, d_out):
    with torch.cuda.stream(stream):
        _train(args, d_out)  # (code and attributes loaded before the capture)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        res = _train(args, d_out)
    return graph, res


def test_graph_keeps_its_scratch():
    """A graph captured on a stream that has a buffer already; then a call there that outgrows that buffer, and tensors
    over the memory it gave back: replays give the same results and leave those tensors alone."""
    args, d_out = _scan_case(6, 700)
    want = [t.clone() for t in _train(args, d_out)]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    graph, res = _capture(stream, args, d_out)
    big, big_do = _scan_case(7, 2100)
    with torch.cuda.stream(stream):
        _train(big, big_do)
        over = [torch.full((1 << 20,), 7, dtype=torch.uint8, device="cuda") for _ in range(64)]
        over += [torch.full((8 << 20,), 7, dtype=torch.uint8, device="cuda") for _ in range(32)]
    torch.cuda.synchronize()
    for _ in range(3):
        for t in res:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for x, y in zip(res, want):
            assert torch.equal(x, y)
    assert all(bool((t == 7).all()) for t in over)


def test_graphs_of_one_stream_side_by_side():
    """Two graphs captured one after the other on the same stream, replayed on two: each has scratch of its own."""
    cases = [_scan_case(s, 900) for s in (8, 9)]
    want = [[t.clone() for t in _train(*c)] for c in cases]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    graphs = [_capture(stream, *c) for c in cases]
    others = [torch.cuda.Stream() for _ in cases]
    for _ in range(20):
        for (graph, _), st in zip(graphs, others):
            with torch.cuda.stream(st):
                graph.replay()
        torch.cuda.synchronize()
        for (_, res), w in zip(graphs, want):
            for x, y in zip(res, w):
                assert torch.equal(x, y)
