"""Norms whose rows stay in registers, at the widths where one form gives way to the next, against the norms in 64 bits."""
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


def near(got, want, rounded, what=""):
    # one rounding to eight bits, or a dozen 32-bit operations and a sum of a few thousand terms
    tol = (2.0 ** -8 if rounded else 4e-6) * max(1.0, float(want.abs().max()))
    err = float((got.cpu().double() - want).abs().max())
    assert err <= tol, f"{what}: {err:.3g} > {tol:.3g}"


def ln(x, w, b=0.0, eps=1e-6):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


WIDTHS = [4, 128, 132, 512, 516, 1024, 1028, 2048, 2052, 4096, 4100]


@pytest.mark.parametrize("H", WIDTHS)
@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("plain", [False, True])
def test_layer_norms(K, H, dtype, plain):
    x, y = rnd(3, H, seed=1) + 40.0, rnd(3, H, seed=2).to(dtype)
    wp, wq, b = rnd(H, seed=3), rnd(H, seed=4), rnd(H, seed=5)
    stream = x.clone().cuda()
    (K.scaled_add(stream, y.cuda(), wp.cuda()) if plain else K.post_norm_add(stream, y.cuda(), wp.cuda(), 1e-6))
    h = K.layernorm(stream, wq.cuda(), 1e-6, dtype, bias=b.cuda())
    want = x.double() + (y.double() * wp.double() if plain else ln(y.double(), wp.double()))
    near(stream, want, False, "stream")
    near(h, ln(want, wq.double(), b.double()), dtype == BF, "norm")


@pytest.mark.parametrize("H", WIDTHS)
def test_mean_of_two_normed_results(K, H):
    a, b, wa, wb, y = rnd(3, H, seed=1), rnd(3, H, seed=2).to(BF), rnd(H, seed=3), rnd(H, seed=4), rnd(3, H, seed=5)
    into = y.clone().cuda()
    K.dual_rmsnorm_mix(a.cuda(), b.cuda(), wa.cuda(), wb.cuda(), 1e-6, 0.5, into)
    K.flush()
    rms = lambda t, w: t.double() / torch.sqrt((t.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    near(into, y.double() + 0.5 * (rms(a, wa) + rms(b, wb)), False)


@pytest.mark.parametrize("S,H", [(1, 128), (2, 132), (3, 512), (4, 516), (4, 1024), (4, 1028), (4, 2048), (4, 2052)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_norm_over_streams_with_an_update(K, S, H, dtype):
    xs, y = rnd(3, S, H, seed=1), rnd(3, H, seed=2).to(dtype)
    mix, out_c, in_c, w = rnd(S, S, seed=3), rnd(S, seed=4), rnd(S, seed=5), rnd(H, seed=6)
    streams = xs.clone().cuda()
    K.streams_update(streams, y.cuda(), mix.cuda(), out_c.cuda())
    h = K.streams_norm(streams, in_c.cuda(), w.cuda(), 1e-6, dtype)
    want = torch.einsum("st,nsh->nth", mix.double(), xs.double()) + out_c.double()[:, None] * y.double()[:, None]
    u = torch.einsum("s,nsh->nh", in_c.double(), want)
    near(streams, want, False, "streams")
    near(h, u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-6) * w.double(), dtype == BF, "norm")


@pytest.mark.parametrize("gs,groups", [(4, 3), (64, 2), (128, 5), (132, 2), (256, 3), (250, 2)])
@pytest.mark.parametrize("mode", ["first", "sigmoid", "silu"])
def test_group_norm_with_gate(K, gs, groups, mode):
    C = gs * groups
    x, gate, w = rnd(5, C, seed=1), rnd(5, C + 4, seed=2).to(BF), rnd(gs, seed=3)
    got = K.group_rmsnorm_gate(x.cuda(), gate.cuda(), 4, w.cuda(), gs, 1e-6, mode == "first", BF, **({} if mode == "first" else {"gate_act": mode}))
    z, v = gate[:, 4:].double(), x.double()
    if mode == "first":
        v = v * torch.nn.functional.silu(z)
    v = v.view(5, groups, gs)
    v = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6) * w.double()).view(5, C)
    v = v if mode == "first" else v * (torch.sigmoid(z) if mode == "sigmoid" else torch.nn.functional.silu(z))
    near(got, v, True)
