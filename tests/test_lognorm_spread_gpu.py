"""GPU tests of the choice between the two tensor-core log-normalisers in the calls that no gradients follow: scores that
the fp16 pairs hold, and sharp ones whose tiles they would mark, which the TF32 kernel takes alone; and the accuracy of
the fp16 pairs on scores just short of that."""
import pytest
import torch

import abi
from transducer_b200 import TransducerLoss
from test_lognorm_f16_gpu import norms, truth

pytestmark = pytest.mark.gpu


def make(B, T, U, V, dtype=torch.float32, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(B + V)
    E = torch.empty((B, T, V), device="cuda").normal_(0, std, generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(0, std, generator=g)
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.randint(T // 2, T + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    ll = torch.randint(U // 2, U, (B,), generator=g, device="cuda", dtype=torch.int32)
    il[0], ll[0] = T, U - 1
    if B > 2:
        il[2] = 0
    return [E, P, labels, il, ll]


def raise_words(E, P, gap, blank=False):
    """One word per frame (or the blank) and another per position `gap` above the rest."""
    g = torch.Generator(device="cuda").manual_seed(7)
    for x, fixed in ((E, blank), (P, False)):
        at = torch.randint(0, x.shape[2], (*x.shape[:2], 1), generator=g, device="cuda")
        if fixed:
            at.zero_()
        x.scatter_add_(2, at, torch.full(at.shape, gap, device="cuda"))


def costs(path, case):
    abi.set_option("lognorm_path", path)
    try:
        with torch.no_grad():
            out = TransducerLoss()(*case)
    finally:
        abi.set_option("lognorm_path", 0)
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(4, 700, 101, 16000), (5, 400, 30, 32000), (64, 500, 21, 2048), (9, 1000, 128, 8192)])
@pytest.mark.parametrize("kind", ["close", "masked", "sharp", "sharp blank", "one sharp utterance"])
def test_which_kernel_takes_the_scores(kind, shape, dtype):
    case = make(*shape)
    E, P = case[:2]
    assert E.numel() > 1 << 25
    if kind == "masked":
        E[:, :, 8:shape[3] // 2] = float("-inf")
        P[:, :, 5:shape[3] // 3] = torch.finfo(torch.float32).min
        case[2].clamp_(max=4)
    elif kind == "one sharp utterance":
        raise_words(E[1:2], P[1:2], 16.0) if shape[0] < 10 else raise_words(E[:16], P[:16], 16.0)
        case[3][1], case[4][1] = shape[1], shape[2] - 1
    elif kind != "close":
        raise_words(E, P, 12.0, kind == "sharp blank")
    case[0], case[1] = E.to(dtype), P.to(dtype)
    auto, tf32, f16 = (costs(path, case) for path in (0, 2, 4))
    assert torch.equal(auto, f16 if kind in ("close", "masked") else tf32)
    assert torch.allclose(f16, tf32, rtol=1e-5)
    if kind == "close":
        assert not torch.equal(f16, tf32)
    assert torch.equal(auto, costs(0, case))


def test_small_calls_stay_with_the_tf32_kernel():
    case = make(8, 500, 51, 8192)
    assert case[0].numel() <= 1 << 25
    assert torch.equal(costs(0, case), costs(2, case))


@pytest.mark.parametrize("gap,std", [(6.0, 1.0), (8.0, 1.0), (9.0, 1.0), (9.5, 1.0), (6.0, 2.0)])
@pytest.mark.parametrize("V", [4096, 16000])
def test_accuracy_of_sharp_scores(V, gap, std):
    """(forced: whatever tile is not marked must be as close to float64 as the TF32 kernel's)"""
    E, P, _, il, ll = make(1, 128, 101, V, std=std)
    raise_words(E, P, gap)
    want = truth(E, P)
    rms = {path: (norms(path, E, P, il, ll)[0].double() - want).pow(2).mean().sqrt().item() for path in (2, 4)}
    assert rms[4] <= rms[2]


def test_a_captured_call_decides_at_every_replay():
    E, P, *rest = make(4, 700, 30, 16000)
    close, sharp = (E, P), (E.clone(), P.clone())
    raise_words(*sharp, 12.0)
    want = [costs(0, [*kind, *rest]) for kind in (close, sharp)]
    held = [E.clone(), P.clone()]
    loss = TransducerLoss(validate_lengths=False)
    stream = torch.cuda.Stream()
    with torch.no_grad(), torch.cuda.stream(stream):
        loss(*held, *rest)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = loss(*held, *rest)
    for i in (0, 1, 0, 1):
        held[0].copy_((close, sharp)[i][0])
        held[1].copy_((close, sharp)[i][1])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[i])
