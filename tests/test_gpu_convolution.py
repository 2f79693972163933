"""The short convolution of prompt portions, four neighbouring channels to a thread, against 64 bits: portions shorter than the taps, around one
chunk of 32 tokens and behind it, one group of channels and more than a block's."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    from llm_infrence_engine_b200.csrc import get_kernels

    return get_kernels()


def step(lens):
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    slots = [len(lens) - 1 - i for i in range(len(lens))]
    return SimpleNamespace(num_seqs=len(lens), max_seq_len=max(lens), seq_starts_dev=torch.tensor(starts, dtype=torch.int32, device="cuda"),
                           seq_slots=torch.tensor(slots, dtype=torch.int32, device="cuda")), starts, slots


def rnd(*shape, seed, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale


@pytest.mark.parametrize("C,act,bias", [(4, None, False), (516, "silu", True)])
def test_short_convolution_of_four_taps(K, C, act, bias):
    lens = [1, 2, 3, 31, 32, 33, 65]
    batch, starts, slots = step(lens)
    z, w, b, st = rnd(starts[-1], C + 8, seed=1).to(BF), rnd(C, 4, seed=2), rnd(C, seed=3) if bias else None, rnd(len(lens), 3, C, seed=4)
    state = st.clone().cuda()
    got = K.causal_conv(z.cuda(), 4, C, w.cuda(), None if b is None else b.cuda(), state, batch, activation=act)
    u = z[:, 4:4 + C].double()
    for r, slot in enumerate(slots):
        rows = torch.cat([st[slot].double(), u[starts[r]:starts[r + 1]]])
        y = sum(rows[j:j + lens[r]] * w[:, j].double() for j in range(4)) + (b.double() if bias else 0.0)
        y = torch.nn.functional.silu(y) if act else y
        err = float((got[starts[r]:starts[r + 1]].cpu().double() - y).abs().max())
        assert err <= 2.0 ** -8 * max(1.0, float(y.abs().max())), (r, err)
        assert torch.equal(state[slot].cpu(), rows[-3:].float())
