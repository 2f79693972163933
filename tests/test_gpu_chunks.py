"""Recurrences that walk sixteen tokens at a time (bfloat16 prompt portions) against the same recurrences token by token in 64 bits: portions around
one and two chunks, states and heads that fill no tile, decays from none to all of a state, and one channel's infinity."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
LENS = [1, 15, 16, 17, 33, 70]


@pytest.fixture(scope="module")
def K():
    from llm_infrence_engine_b200.csrc import get_kernels

    return get_kernels()


@pytest.fixture(autouse=True)
def always(K):
    before = K.chunk_scan_rows, K.chunk_scan_blocks
    K.chunk_scan_rows, K.chunk_scan_blocks = (1, 1, 1), (1e9, 1e9, 1e9)
    yield
    K.chunk_scan_rows, K.chunk_scan_blocks = before


def step(lens):
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    slots = [len(lens) - 1 - i for i in range(len(lens))]
    return SimpleNamespace(num_seqs=len(lens), max_seq_len=max(lens), seq_starts_dev=torch.tensor(starts, dtype=torch.int32, device="cuda"),
                           seq_slots=torch.tensor(slots, dtype=torch.int32, device="cuda")), starts, slots


def rnd(*shape, seed, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale


def near(got, want, what):
    # rounding of a few hundred 32-bit operations, each of the size of the result
    err = float((got.cpu().double() - want).abs().max()) / max(1.0, float(want.abs().max()))
    assert err <= 3e-5, f"{what}: {err:.3g}"


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("H,G,D,DV", [(3, 1, 24, 20), (2, 2, 64, 16), (4, 2, 100, 36), (2, 1, 128, 130)])
def test_delta_rule(K, H, G, D, DV, per_head):
    batch, starts, slots = step(LENS)
    N, DA = starts[-1], 1 if per_head else D
    qkv, a, b = rnd(N, 2 * G * D + H * DV, seed=1).to(BF), (rnd(N, H * DA, seed=2) * 6).to(BF), rnd(N, H, seed=3).to(BF)
    A_log, dt_bias, st = rnd(H, seed=4) * 2, rnd(H * DA, seed=5) - 3, rnd(len(LENS), H, DV, D, seed=6, scale=0.1)
    state = st.clone().cuda()
    got = K.delta_rule(qkv.cuda(), H, G, D, DV, a.cuda(), b.cuda(), 0, A_log.cuda(), dt_bias.cuda(), state, batch, decay_per_head=per_head)
    q, k, v = qkv.double().split([G * D, G * D, H * DV], 1)
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q, k, v = unit(q.view(N, G, D)) * D ** -0.5, unit(k.view(N, G, D)), v.view(N, H, DV)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    decay = torch.exp(-torch.exp(A_log.double())[:, None] * torch.nn.functional.softplus((a.double() + dt_bias.double()).view(N, H, DA)))
    want, S = torch.zeros(N, H, DV, dtype=torch.float64), st.double()
    for r, slot in enumerate(slots):
        s = S[slot].transpose(1, 2).clone()
        for t in range(starts[r], starts[r + 1]):
            s = decay[t][:, :, None] * s
            u = torch.sigmoid(b[t].double())[:, None] * (v[t] - (k[t][:, None] @ s)[:, 0])
            s = s + k[t][:, :, None] * u[:, None]
            want[t] = (q[t][:, None] @ s)[:, 0]
        S[slot] = s.transpose(1, 2)
    near(got, want.view(N, -1), "outputs")
    near(state, S, "states")


@pytest.mark.parametrize("H,G,NS,DV", [(6, 2, 20, 12), (2, 1, 64, 16), (4, 4, 128, 34)])
def test_state_space(K, H, G, NS, DV):
    batch, starts, slots = step(LENS)
    N = starts[-1]
    x, dt = rnd(N, H * DV + 2 * G * NS, seed=1).to(BF), (rnd(N, H, seed=2) * 4).to(BF)
    A_log, bias, skip, st = rnd(H, seed=3), rnd(H, seed=4) - 2, rnd(H, seed=5), rnd(len(LENS), H, DV, NS, seed=6, scale=0.1)
    state = st.clone().cuda()
    got = K.ssm_scan(x.cuda(), H, G, NS, DV, dt.cuda(), 0, A_log.cuda(), bias.cuda(), skip.cuda(), state, batch)
    u, B, C = x.double().split([H * DV, G * NS, G * NS], 1)
    u, B, C = u.view(N, H, DV), B.view(N, G, NS).repeat_interleave(H // G, 1), C.view(N, G, NS).repeat_interleave(H // G, 1)
    d = torch.nn.functional.softplus(dt.double() + bias.double())
    a = torch.exp(-torch.exp(A_log.double()) * d)
    want, S = torch.zeros(N, H, DV, dtype=torch.float64), st.double()
    for r, slot in enumerate(slots):
        s = S[slot].transpose(1, 2).clone()
        for t in range(starts[r], starts[r + 1]):
            s = a[t][:, None, None] * s + (d[t][:, None] * B[t])[:, :, None] * u[t][:, None]
            want[t] = (C[t][:, None] @ s)[:, 0] + skip.double()[:, None] * u[t]
        S[slot] = s.transpose(1, 2)
    near(got, want.view(N, -1), "outputs")
    near(state, S, "states")


def test_an_infinity_stays_behind_its_token(K):
    """What follows in the same chunk may be lost, what came before must not be, nor the columns beside."""
    batch, starts, _ = step([24])
    x, dt = rnd(24, 2 * 16 + 2 * 32, seed=1).to(BF), rnd(24, 2, seed=2).to(BF)
    args = [t.cuda() for t in (rnd(2, seed=3), rnd(2, seed=4), rnd(2, seed=5))]
    clean = K.ssm_scan(x.cuda(), 2, 1, 32, 16, dt.cuda(), 0, *args, torch.zeros(1, 2, 16, 32, device="cuda"), batch)
    x[9, 5] = float("inf")
    got = K.ssm_scan(x.cuda(), 2, 1, 32, 16, dt.cuda(), 0, *args, torch.zeros(1, 2, 16, 32, device="cuda"), batch)
    assert torch.equal(got[:9], clean[:9]) and not bool(torch.isfinite(got[9, 5]))
    others = [c for c in range(32) if c != 5]
    assert torch.equal(got[:, others], clean[:, others])
