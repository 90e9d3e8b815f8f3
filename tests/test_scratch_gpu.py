"""The zero-filled scratch of split rows: whose it is in plain stream order, under stream capture, and when it goes back."""
import gc
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

B, L, K = 2, 1 << 20, 512


def _rows(seed):
    from flash_float_jit_kernels_b200 import workloads
    s, lengths, _ = workloads.gaussian_bf16_ties(B, L, seed=seed)
    return s, lengths


def _capture(side, s, lengths, out, **kw):
    from flash_float_jit_kernels_b200 import fast_topk_v3
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side, **kw):
        fast_topk_v3(s, lengths, K, out=out)
    return graph


def test_the_shape_is_one_that_uses_scratch():
    import ctypes
    from flash_float_jit_kernels_b200 import _lib
    lib = _lib.load()
    shape = (ctypes.c_int32 * 2)()
    assert lib.ff_topk_policy_launch_shape(B, L, K, 1, 0, shape) == 0 and shape[1] > 1
    assert lib.ff_topk_workspace_bytes(B, L, K) > 0


def test_second_graph_of_a_fresh_stream_needs_no_replay_of_the_first(oracle):
    """Two selects captured on a stream that never ran one, out of a memory pool whose free blocks hold garbage: the
    second graph and an eager call on the stream find zeroed scratch although the first graph never ran."""
    from flash_float_jit_kernels_b200 import fast_topk_v3
    dev = torch.device("cuda:0")
    (s1, lengths), (s2, _) = _rows(1), _rows(2)
    d1, d2, ld = s1.to(dev), s2.to(dev), lengths.to(dev)
    fast_topk_v3(d1, ld, K)                                  # one-time set-up, on another stream
    torch.cuda.synchronize()
    side, pool = torch.cuda.Stream(), torch.cuda.graph_pool_handle()
    dirty = torch.cuda.CUDAGraph()
    with torch.cuda.graph(dirty, stream=side, pool=pool):
        garbage = torch.full((64 << 20,), 0xAB, dtype=torch.uint8, device=dev)
    dirty.replay()
    torch.cuda.synchronize()
    del garbage                                              # its block is free in the pool now
    o1, o2 = (torch.empty((B, K), dtype=torch.int32, device=dev) for _ in range(2))
    g1 = _capture(side, d1, ld, o1, pool=pool)
    g2 = _capture(side, d2, ld, o2, pool=pool)
    g2.replay()
    with torch.cuda.stream(side):
        eager = fast_topk_v3(d1, ld, K)
    torch.cuda.synchronize()
    assert np.array_equal(o2.cpu().numpy(), oracle.topk_c(s2.numpy(), lengths.numpy(), K))
    exp1 = oracle.topk_c(s1.numpy(), lengths.numpy(), K)
    assert np.array_equal(eager.cpu().numpy(), exp1)
    g1.replay()
    torch.cuda.synchronize()
    assert np.array_equal(o1.cpu().numpy(), exp1)
    del g1, g2, dirty


def test_graphs_of_one_stream_replayed_on_two(oracle):
    """Graphs captured one after the other on one stream share no scratch, so their replays may overlap."""
    dev = torch.device("cuda:0")
    rows = [_rows(3), _rows(4)]
    side = torch.cuda.Stream()
    data = [(s.to(dev), l.to(dev), torch.empty((B, K), dtype=torch.int32, device=dev)) for s, l in rows]
    torch.cuda.synchronize()
    graphs = [_capture(side, *d) for d in data]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
    torch.cuda.synchronize()
    for (s, l), (_, _, out) in zip(rows, data):
        assert np.array_equal(out.cpu().numpy(), oracle.topk_c(s.numpy(), l.numpy(), K))
    del graphs, graph


def test_scratch_of_many_captures_is_bounded_and_goes_back():
    """The first captures keep their buffers, up to a bound; those of later ones go back with their graphs."""
    from flash_float_jit_kernels_b200 import _host, _lib, fast_topk_v3
    dev = torch.device("cuda:0")
    s, lengths = _rows(5)
    d, ld, out = s.to(dev), lengths.to(dev), torch.empty((B, K), dtype=torch.int32, device=dev)
    side = torch.cuda.Stream()
    fast_topk_v3(d, ld, K, out=out)                          # the current stream's own buffer
    _capture(side, d, ld, out)                               # (the side stream's handles and pools)
    gc.collect()

    def settled():
        for _ in range(50):                                  # the runtime gives a buffer back on a thread of its own
            torch.cuda.synchronize()
            _host.scratch()(0, 256)
            time.sleep(0.01)
        return torch.cuda.memory_allocated()

    bound, need = 64 << 20, int(_lib.load().ff_topk_workspace_bytes(B, L, K))
    before = settled()
    for _ in range(bound // need + 1):
        _capture(side, d, ld, out)
    gc.collect()
    kept = settled()
    assert kept - before <= bound + (2 << 20)
    graphs = [_capture(side, d, ld, out) for _ in range(8)]
    assert torch.cuda.memory_allocated() - kept >= 8 * need
    for g in graphs:
        g.replay()
    torch.cuda.synchronize()
    del graphs, g
    gc.collect()
    assert settled() == kept
