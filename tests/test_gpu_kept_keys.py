"""Kept first tokens and a query temperature on the tcgen05 attention of prompt portions, and the temperature on the decode kernel, against the
plain statement: kept keys that end inside, at and behind a chunk's edge, portions before, across and far behind the window's end."""
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


VARIANTS = {"kept 4": dict(window=136, keep_first=4), "kept a chunk": dict(window=70, keep_first=64), "kept more": dict(window=9, keep_first=131),
            "kept within the window": dict(window=700, keep_first=3), "kept and cap": dict(window=64, keep_first=20, softcap=2.0),
            "temperature": dict(temp=(0.4, 16)), "temperature and cap": dict(temp=(0.3, 7), softcap=1.5), "temperature, window, kept": dict(temp=(0.4, 16), window=100, keep_first=5)}


@pytest.mark.parametrize("nq,nkv,d,page", [(4, 1, 64, 16), (14, 2, 64, 8), (4, 2, 128, 64)])
@pytest.mark.parametrize("first,n", [(0, 300), (37, 200), (640, 90)])
@pytest.mark.parametrize("what", list(VARIANTS))
def test_prompt_portions(K, nq, nkv, d, page, first, n, what):
    kw = dict(VARIANTS[what])
    window = kw.pop("window", 0)
    ctx_len = first + n
    k_pool, v_pool, table, _, _ = paged(ctx_len, page, nkv, d, d, "bfloat16", 3)
    k_pool[0], v_pool[0] = float("nan"), float("nan")
    pos, seq = torch.arange(first, ctx_len, dtype=torch.int32), torch.ones(n, dtype=torch.int32)
    q = rnd(n, nq * d, seed=5, scale=0.5).bfloat16()
    want = TorchKernels().attention_ext(q, 0, nq, nkv, d, d, k_pool, v_pool, table, seq, pos, page, 0.3, window, ctx_len, **kw)
    batch = SimpleNamespace(seq_lens=[n], seq_starts_dev=torch.tensor([0, n], dtype=torch.int32).cuda(), max_seq_len=n, num_seqs=1, _tables={})
    args = [t.cuda() for t in (k_pool, v_pool, table, seq, pos)]
    for more in ({}, {"num_splits": 3}):
        calls = []
        plain, K._attention_tc = K._attention_tc, lambda *a, **k: calls.append(1) or plain(*a, **k)
        try:
            got = K.attention_ext(q.cuda(), 0, nq, nkv, d, d, *args, page, 0.3, window, ctx_len, batch=batch, **kw, **more)
        finally:
            del K._attention_tc
        assert calls
        close(got, want, "bfloat16", f"{what} {more}")
    K.check_device_errors()


@pytest.mark.parametrize("nq,nkv,d", [(4, 1, 64), (14, 2, 64), (4, 2, 128)])
def test_temperature_of_decoded_tokens(K, nq, nkv, d):
    ctx_len, page = 1300, 16
    k_pool, v_pool, table, _, _ = paged(ctx_len, page, nkv, d, d, "bfloat16", 3)
    pos = torch.tensor([0, 1, 15, 16, 255, 256, 1299], dtype=torch.int32)
    n = pos.shape[0]
    seq, q, gate = torch.ones(n, dtype=torch.int32), rnd(n, nq * d, seed=5, scale=0.5).bfloat16(), rnd(n, nq, seed=6).bfloat16()
    batch = SimpleNamespace(seq_lens=[1] * n, seq_starts_dev=torch.arange(n + 1, dtype=torch.int32).cuda(), max_seq_len=1, num_seqs=n, _tables={})
    for kw in (dict(temp=(0.4, 16)), dict(temp=(0.4, 16), softcap=1.5, gate=gate, gate_per_head=True)):
        want = TorchKernels().attention_ext(q, 0, nq, nkv, d, d, k_pool, v_pool, table, seq, pos, page, 0.3, 0, ctx_len, **kw)
        got = K.attention_ext(q.cuda(), 0, nq, nkv, d, d, k_pool.cuda(), v_pool.cuda(), table.cuda(), seq.cuda(), pos.cuda(), page, 0.3, 0, ctx_len,
                              batch=batch, **{k: v.cuda() if isinstance(v, torch.Tensor) else v for k, v in kw.items()})
        close(got, want, "bfloat16", str(list(kw)))
