"""Calls on several streams and from several threads: the cached scratch of one is not touched by another."""
import threading

import pytest
import torch

from mixlab_b200 import ops
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
