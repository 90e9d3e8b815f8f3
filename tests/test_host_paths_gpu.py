"""The native host path of the operators and the Python layer behind it make the same call: every form once through each
(a tensor subclass is what the native path leaves to Python)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


class _Subclass(torch.Tensor):
    pass


def _wrapped(t):
    return t.as_subclass(_Subclass)


@pytest.mark.parametrize("B,L", [(1, 1 << 20), (3, 20000), (64, 9000), (200, 4001)])
@pytest.mark.parametrize("form", ["plain", "int64", "bf16", "f16", "windows", "out", "guesses", "columns of a wider buffer"])
def test_select(B, L, form):
    from flash_float_jit_kernels_b200 import _host, fast_topk_v3, new_threshold_hint
    g = torch.Generator(device=DEV).manual_seed(L)
    k = 300
    s = torch.randn((B, L), generator=g, device=DEV)
    lengths = torch.randint(1, L + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    rs, kw = None, {}
    if form in ("bf16", "f16"):
        s = s.to(torch.bfloat16 if form == "bf16" else torch.float16)
    if form == "int64":
        kw["index_dtype"] = torch.int64
    if form == "windows":
        rs = torch.randint(0, 60, (B,), generator=g, device=DEV, dtype=torch.int32)
        lengths = torch.minimum(lengths, L - rs)
    if form == "columns of a wider buffer":
        s = torch.randn((B, L + 37), generator=g, device=DEV)[:, 5:5 + L]
    results = []
    for wrap in (lambda t: t, _wrapped):
        if form == "out":
            kw["out"] = torch.empty((B, k), device=DEV, dtype=torch.int32)
        if form == "guesses":
            kw["threshold_hint"] = new_threshold_hint(B, DEV)
        for _ in range(2 if form == "guesses" else 1):
            r = fast_topk_v3(wrap(s), lengths, k, rs, **kw)
        if form == "out":
            assert r is kw["out"]
        results.append((r.cpu().numpy(), kw["threshold_hint"].cpu().numpy() if form == "guesses" else None))
    assert _host.topk()(_wrapped(s), lengths, k, rs, None, None, None, torch.int32, None) is None
    (a, ha), (b, hb) = results
    assert a.dtype == b.dtype and np.array_equal(a, b)
    if ha is not None:
        assert np.array_equal(np.isnan(ha), np.isnan(hb))


@pytest.mark.parametrize("B,L,requests", [(5, 30000, 5), (40, 6000, 3), (2, 300000, 2)])
def test_transforms(B, L, requests):
    from flash_float_jit_kernels_b200 import fast_topk_transform_fused, fast_topk_transform_ragged_fused
    g = torch.Generator(device=DEV).manual_seed(B)
    k = 512
    s = torch.randn((B, L), generator=g, device=DEV)
    lengths = torch.randint(1, L + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    table = torch.randint(0, 1 << 20, (requests, L), generator=g, device=DEV, dtype=torch.int32)
    cu = torch.tensor([B * i // requests for i in range(requests + 1)], device=DEV, dtype=torch.int32)
    offset = torch.arange(B, device=DEV, dtype=torch.int32) * 1000
    outs = []
    for wrap in (lambda t: t, _wrapped):
        pages, ragged = (torch.empty((B, k), device=DEV, dtype=torch.int32) for _ in range(2))
        fast_topk_transform_fused(wrap(s), lengths, pages, table, cu)
        fast_topk_transform_ragged_fused(wrap(s), lengths, ragged, offset)
        outs.append((pages.cpu().numpy(), ragged.cpu().numpy()))
    assert all(np.array_equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("B,L", [(3, 5000), (1100, 200)])
def test_logits(B, L):
    from flash_float_jit_kernels_b200 import fast_topk_v3
    from flash_float_jit_kernels_b200.indexer_logits import indexer_logits_fp8, new_handover
    g = torch.Generator(device=DEV).manual_seed(B)
    q = (torch.randn((B, 64, 128), generator=g, device=DEV) / 4).to(torch.float8_e4m3fn)
    keys = (torch.randn((B, L, 128), generator=g, device=DEV) / 4).to(torch.float8_e4m3fn)
    w = torch.rand((B, 64), generator=g, device=DEV)
    lengths = torch.randint(0, L + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    outs = []
    for wrap in (lambda t: t, _wrapped):
        hint, handover = torch.zeros((B,), device=DEV), new_handover(B, DEV)
        fresh = indexer_logits_fp8(q, keys, wrap(w), lengths)
        kept = torch.full((B, L), 3.0, device=DEV)
        assert indexer_logits_fp8(q, keys, wrap(w), lengths, out=kept, threshold_hint=hint, handover=handover) is kept
        picked = fast_topk_v3(wrap(fresh), lengths, 100, threshold_hint=hint, handover=handover)
        outs.append([t.cpu().numpy() for t in (fresh, kept, picked)])
    assert all(np.array_equal(a, b) for a, b in zip(*outs))
