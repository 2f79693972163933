"""Keys of talking heads in slices (prompt portions, and shorter ones for decoded tokens) against the plain statement, with slices that no token, some
tokens or all tokens of a tile see; and the layout of the chosen experts' runs and tiles at the edges of a warp's lanes."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from test_gpu_zepalorn import close, paged, rnd
from torch_kernels import TorchKernels

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from llm_infrence_engine_b200.csrc import get_kernels

    return get_kernels()


@pytest.mark.parametrize("nq,nkv,d", [(8, 2, 128), (16, 4, 64), (4, 2, 32), (6, 3, 64)])
@pytest.mark.parametrize("first,n", [(0, 100), (70, 65), (0, 3)])
@pytest.mark.parametrize("chunks", [1, 2])
def test_talking_heads_in_slices(K, nq, nkv, d, first, n, chunks):
    ctx_len, page = first + n, 16
    k_pool, v_pool, table, _, _ = paged(ctx_len, page, nkv, d, d, "bfloat16", 3)
    pos, seq = torch.arange(first, ctx_len, dtype=torch.int32), torch.ones(n, dtype=torch.int32)
    q, talk, sink, gate = rnd(n, nq * d, seed=5, scale=0.5).bfloat16(), rnd(nq, nq, seed=6, scale=0.5), rnd(nq, seed=7), rnd(n, nq, seed=8).bfloat16()
    kw = dict(talk=talk, sink=sink, gate=gate, gate_per_head=True, softcap=5.0)
    want = TorchKernels().attention_ext(q, 0, nq, nkv, d, d, k_pool, v_pool, table, seq, pos, page, 0.2, 0, ctx_len, **kw)
    dev = {k: v.cuda() if isinstance(v, torch.Tensor) else v for k, v in kw.items()}
    args = [t.cuda() for t in (k_pool, v_pool, table, seq, pos)]
    portion = SimpleNamespace(seq_lens=[n], seq_starts_dev=torch.tensor([0, n], dtype=torch.int32).cuda(), max_seq_len=n, num_seqs=1, _tables={})
    K.talk_slice_chunks, before = chunks, K.talk_slice_chunks
    try:
        got = K.attention_ext(q.cuda(), 0, nq, nkv, d, d, *args, page, 0.2, 0, ctx_len, batch=portion, **dev)
    finally:
        K.talk_slice_chunks = before
    close(got, want, "bfloat16", "prompt portion")
    single = SimpleNamespace(seq_lens=[1] * n, seq_starts_dev=torch.arange(n + 1, dtype=torch.int32).cuda(), max_seq_len=1, num_seqs=n, _tables={})
    for short in (True, False):
        K.short_talk_slices = short
        try:
            got = K.attention_ext(q.cuda(), 0, nq, nkv, d, d, *args, page, 0.2, 0, ctx_len, batch=single, **dev)
        finally:
            K.short_talk_slices = True
        close(got, want, "bfloat16", f"single tokens, short slices {short}")


@pytest.mark.parametrize("pairs,E,tile_rows", [(1, 1, 4), (32, 16, 4), (64, 31, 1), (200, 32, 128), (513, 33, 4), (700, 65, 2), (40, 300, 4)])
def test_layout_of_the_chosen_experts(K, pairs, E, tile_rows):
    ids = torch.randint(0, E + 2, (pairs,), generator=torch.Generator().manual_seed(pairs), dtype=torch.int32)   # (from E on: identity experts)
    ids[: pairs // 2] = ids[: pairs // 2].clamp(max=max(0, E // 3))   # some experts with several tiles, some with none
    most = -(-pairs // tile_rows) + E
    offsets, perm, place, tiles = (torch.full((n,), -7, dtype=torch.int32, device="cuda") for n in (E + 1, pairs, pairs, 1 + 2 * most))
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    dev_ids = ids.cuda()
    assert K.lib.llmie_moe_sort(p(dev_ids), pairs, E, tile_rows, p(offsets), p(perm), p(place), p(tiles), most, K._stream()) == 0
    counts = [int((ids == e).sum()) for e in range(E)]
    starts = [sum(counts[:e]) for e in range(E + 1)]
    assert offsets.tolist() == starts
    want = [(e, starts[e] + r) for e in range(E) for r in range(0, counts[e], tile_rows)]
    flat = tiles.tolist()
    assert flat[0] == len(want) and list(zip(flat[1::2], flat[2::2]))[: len(want)] == want
    for i, (e, at) in enumerate(zip(ids.tolist(), place.tolist())):
        assert (at == -1) if e >= E else (starts[e] <= at < starts[e + 1] and int(perm[at]) == i)
