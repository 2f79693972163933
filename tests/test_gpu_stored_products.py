"""The small-batch product whose result is stored (the blocks that share K form a cluster), at the edges of its tiles: rows and outputs that fill
none or part of a tile, K of one piece and of more pieces than blocks, columns of wider rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    from llm_infrence_engine_b200.csrc import get_kernels

    return get_kernels()


def rnd(*shape, seed, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale


@pytest.mark.parametrize("M,N,Kd", [(1, 8, 8), (16, 128, 64), (17, 130, 520), (33, 100, 72), (64, 257, 200), (65, 64, 1032), (128, 24, 136)])
def test_stored_product(K, M, N, Kd):
    x, w = rnd(M, Kd, seed=M).to(BF), rnd(N, Kd, seed=N, scale=Kd ** -0.5).to(BF)
    want = x.double() @ w.double().T
    scale = float(want.abs().max())
    blocks = 1
    while blocks <= min(8, -(-Kd // 64)):
        for out in (BF, torch.float32):
            got = K.linear_tc_store(x.cuda(), w.cuda(), out, blocks=blocks)
            # a rounding to eight bits (2^-9 of the value), or sums of Kd exact products in 32 bits
            tol = 2.0 ** -8 * scale if out == BF else 1e-6 * Kd ** 0.5 * max(1.0, scale)
            assert got.dtype == out and float((got.cpu().double() - want).abs().max()) <= tol, (blocks, out)
        blocks *= 2
    K.check_device_errors()


def test_bias_and_columns_of_wider_rows(K):
    wide, w, b = rnd(5, 300, seed=1).to(BF), rnd(70, 64, seed=2, scale=0.1).to(BF), rnd(70, seed=3).to(BF)
    x = wide.cuda()[:, 24:88]   # rows 600 bytes apart: not a multiple of 16, the library's product
    aligned = torch.nn.functional.pad(wide, (0, 4)).cuda()[:, 24:88]
    want = wide[:, 24:88].double() @ w.double().T + b.double()
    for at in (x, aligned):
        got = K.linear(at, w.cuda(), bias=b.cuda())
        assert float((got.cpu().double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    assert aligned.stride(0) % 8 == 0 and K._stored_by_tc(aligned, w.cuda()) and not K._stored_by_tc(x, w.cuda())
