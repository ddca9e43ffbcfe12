"""GPU tests of how the tensor-core gradient kernel goes through an utterance's frames: halves of a tile or alternate
tiles, whole items or cut ones, on both sides of each rule, in both storage types and in place."""
import pytest
import torch

import abi

pytestmark = pytest.mark.gpu

# utterances, frames, positions, words: 48 frames a tile for 65..112 positions, 64 below, 32 above
SHAPES = [
    # 80 items, not cut.  Halves (up to five tiles), then alternate tiles: their first, a ring of four stages gone through
    # several times, odd and even numbers of tiles
    (8, 240, 101, 1280), (8, 241, 101, 1280), (8, 288, 101, 1280), (8, 700, 101, 1280), (8, 768, 70, 1280),
    (8, 700, 50, 1280), (8, 700, 128, 1280),
    # 64 items, in two parts from 576 frames on
    (8, 575, 101, 1000), (8, 576, 101, 1000), (8, 1500, 101, 1000), (8, 700, 30, 1000),
    # few items: from 288 frames on, up to 16 parts
    (3, 287, 80, 104), (3, 288, 80, 104), (2, 2000, 101, 64),
]


def make(B, T, U, V, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(B + T + U + V)
    E = torch.empty((B, T, V), device="cuda").normal_(0, 1, generator=g).to(dtype)
    P = torch.empty((B, U, V), device="cuda").normal_(0, 1, generator=g).to(dtype)
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.randint(T // 2, T + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    ll = torch.randint(U // 2, U, (B,), generator=g, device="cuda", dtype=torch.int32)
    il[0], ll[0] = T, U - 1
    for b, t in enumerate((1, 49, 240, 288, 0), 2):   # (short ones beside the long ones)
        if b < B:
            il[b] = min(t, T)
    return E, P, labels, il, ll, torch.linspace(0.5, 1.5, B, device="cuda")


def grads(E, P, labels, il, ll, deltas, path=0):
    abi.set_option("grads_path", path)
    try:
        fwd = abi.loss_forward(E, P, labels, il, ll)
        eg, pg = abi.loss_backward(E, P, labels, il, ll, fwd, deltas)
        torch.cuda.synchronize()
    finally:
        abi.set_option("grads_path", 0)
    abi.check(abi.lib.tb200_check_status())
    return fwd, eg, pg


@pytest.mark.parametrize("shape", SHAPES)
def test_against_the_simt_kernels(shape):
    case = make(*shape)
    _, eg_s, pg_s = grads(*case, path=1)
    _, eg, pg = grads(*case, path=2)
    # (the bar of the other tests of this kernel: exp(E) in two TF32 halves, exp(P) in one)
    assert (eg - eg_s).abs().max().item() <= 1e-3 * eg_s.abs().max().item()
    assert (pg - pg_s).abs().max().item() <= 1e-3 * pg_s.abs().max().item()
    for b in range(shape[0]):
        assert not eg[b, int(case[3][b]):].any() and not pg[b, int(case[4][b]) + 1:].any()


@pytest.mark.parametrize("shape", SHAPES)
def test_bf16_storage(shape):
    """The fp32 results rounded once to bf16, one unit of slack; where a block of 128 columns holds more than 16 labels their
    terms come off the rounded number, one unit of the largest entry."""
    E, P, *rest = make(*shape, dtype=torch.bfloat16)
    _, eg, pg = grads(E, P, *rest)
    _, eg32, pg32 = grads(E.float(), P.float(), *rest)
    for got, ref in ((eg, eg32), (pg, pg32)):
        want = ref.bfloat16().float()
        ulp = torch.maximum(want.abs(), ref.abs()) * 2.0 ** -7 + 1e-30
        if got is eg:
            ulp = ulp + ref.abs().max() * 2.0 ** -8
        assert bool(((got.float() - want).abs() <= ulp).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(8, 700, 101, 1280), (8, 700, 101, 1000), (3, 300, 80, 104), (2, 2000, 128, 64)])
def test_in_place(shape, dtype):
    """Over emissions and predictions: bit for bit the same, where the frames of an item are in several CTAs too."""
    B, T, U, V = shape
    E, P, labels, il, ll, deltas = make(*shape, dtype=dtype)
    fwd, eg, pg = grads(E, P, labels, il, ll, deltas)
    n = abi.lib.tb200_loss_backward_workspace_bytes(B, T, U, V)
    ws = abi.workspace(n)
    fn = abi.lib.tb200_loss_backward_bf16 if dtype is torch.bfloat16 else abi.lib.tb200_loss_backward
    abi.use_torch_stream()
    abi.check(fn(abi.ptr(E), abi.ptr(P), abi.ptr(labels), abi.ptr(il), abi.ptr(ll), abi.ptr(fwd["saved"]),
                 fwd["saved"].numel(), abi.ptr(deltas), abi.ptr(E), abi.ptr(P), B, T, U, V, 0, abi.ptr(ws), n))
    torch.cuda.synchronize()
    assert torch.equal(E.view(torch.uint8), eg.view(torch.uint8))
    assert torch.equal(P.view(torch.uint8), pg.view(torch.uint8))
