"""Rows split over single CTAs, which are launched without the promise that they run together: exact whoever gives a wait for the
others up, and nothing left in the scratch."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib():
    from flash_float_jit_kernels_b200 import _lib
    lib = _lib.load()
    yield lib
    lib.ff_topk_set_wait_limit(0)


def _rows(kind, B, L, seed):
    g = torch.Generator().manual_seed(seed)
    s = torch.randn((B, L), generator=g)
    if kind == "ties":
        s = s.to(torch.bfloat16).float()
    elif kind == "sorted":                       # its own guess does not fit: the histogram path
        s = torch.sort(s, dim=1).values
    elif kind == "equal":                        # all digit levels
        s = torch.full((B, L), 3.0)
    lengths = torch.full((B,), L, dtype=torch.int32)
    if B > 1:
        lengths[1] = L - 12345
    return s, lengths


@pytest.mark.parametrize("polls", [1, 2, 6, 40])
@pytest.mark.parametrize("kind,dtype", [("normal", torch.float32), ("ties", torch.bfloat16), ("sorted", torch.float32),
                                        ("equal", torch.float32), ("normal", torch.float16)])
@pytest.mark.parametrize("B,L,k", [(1, 1 << 20, 2048), (3, 900_001, 512)])
def test_a_row_whose_ctas_give_up_is_exact(lib, oracle, polls, kind, dtype, B, L, k):
    from flash_float_jit_kernels_b200 import fast_topk_v3, new_threshold_hint
    shape = (ctypes.c_int32 * 2)()
    assert lib.ff_topk_policy_launch_shape(B, L, k, 1, 0, shape) == 0 and shape[0] == 1 and shape[1] > 1
    dev = torch.device("cuda:0")
    s, lengths = _rows(kind, B, L, polls)
    s = s.to(dtype)
    exp = oracle.topk_c(s.float().numpy(), lengths.numpy(), k)
    sd, ld = s.to(dev), lengths.to(dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    hint = new_threshold_hint(B, dev)
    for limit in (polls, 0, polls, polls, 0):    # given up or not, in turn: what one leaves in the scratch the next one finds
        lib.ff_topk_set_wait_limit(limit)
        assert np.array_equal(fast_topk_v3(sd, ld, k, status=status).cpu().numpy(), exp)
        assert np.array_equal(fast_topk_v3(sd, ld, k, status=status, threshold_hint=hint).cpu().numpy(), exp)
    assert int(status.item()) & ~8 == 0          # (8: a caller's guess did not fit)


def test_several_streams_at_once(lib, oracle):
    from flash_float_jit_kernels_b200 import fast_topk_v3
    dev, k, n = torch.device("cuda:0"), 2048, 4
    rows = [_rows("normal", 1, (1 << 20) + 77 * i, i) for i in range(n)]
    exp = [oracle.topk_c(s.numpy(), l.numpy(), k) for s, l in rows]
    rows = [(s.to(dev), l.to(dev)) for s, l in rows]
    streams = [torch.cuda.Stream(priority=-(i % 2)) for i in range(n)]
    torch.cuda.synchronize()
    outs = [[] for _ in range(n)]
    for _ in range(8):
        for i in range(n):
            with torch.cuda.stream(streams[i]):
                outs[i].append(fast_topk_v3(*rows[i], k))
    torch.cuda.synchronize()
    for i in range(n):
        assert all(np.array_equal(o.cpu().numpy(), exp[i]) for o in outs[i])


def test_replays_give_up_too(lib, oracle):
    from flash_float_jit_kernels_b200 import fast_topk_v3
    dev, k = torch.device("cuda:0"), 1024
    s, lengths = _rows("normal", 2, 1 << 20, 5)
    exp = oracle.topk_c(s.numpy(), lengths.numpy(), k)
    sd, ld = s.to(dev), lengths.to(dev)
    out = torch.empty((2, k), dtype=torch.int32, device=dev)
    fast_topk_v3(sd, ld, k, out=out)
    lib.ff_topk_set_wait_limit(2)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fast_topk_v3(sd, ld, k, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), exp)
