"""GPU tests of the log-normaliser on fp16 pairs: edges of its stages (64 words), tiles (128 frames) and column
ranges (160 positions) against float64, its distance to float64 against the TF32 kernel's, and inputs beyond
the range of fp16, whose tiles the TF32 kernel has to take over."""
import pytest
import torch

import abi

pytestmark = pytest.mark.gpu


def norms(path, E, P, il, ll):
    abi.set_option("lognorm_path", path)
    try:
        out = abi.log_norms(E, P, il, ll)
        torch.cuda.synchronize()
    finally:
        abi.set_option("lognorm_path", 0)
    return out


def truth(E, P):
    return torch.stack([torch.cat([torch.logsumexp(e[t:t + 16, None].double() + p[None].double(), 2)
                                   for t in range(0, e.shape[0], 16)]) for e, p in zip(E, P)])


def make(B, T, U, V, std=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    E = torch.empty((B, T, V), device="cuda").normal_(0, std, generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(0, std, generator=g)
    il = torch.randint(1, T + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    ll = torch.randint(0, U, (B,), generator=g, device="cuda", dtype=torch.int32)
    il[0], ll[0] = T, U - 1
    return E, P, il, ll


def valid(il, ll, T, U):
    return torch.as_tensor(abi.valid_mask(il.cpu().numpy(), ll.cpu().numpy(), T, U), device="cuda")


@pytest.mark.parametrize("V", [32, 36, 60, 64, 68, 96, 124, 128, 132, 196, 1000])
@pytest.mark.parametrize("T,U", [(1, 1), (127, 16), (128, 17), (129, 112), (140, 120), (33, 121), (130, 128),
                                 (20, 129), (50, 144), (40, 145), (130, 160), (129, 161), (30, 208), (129, 256)])
def test_edges_against_float64(T, U, V):
    E, P, il, ll = make(3, T, U, V, std=1.5, seed=T + U + V)
    ln, ref, mp = norms(4, E, P, il, ll)
    _, ref2, mp2 = norms(2, E, P, il, ll)
    m = valid(il, ll, T, U)
    want = truth(E, P)
    # 22 bits a factor and the marks' 2^-20 at worst, an fp32 logarithm and two additions at LN's magnitude
    tol = 2.0 ** -20 + 4 * 2.0 ** -23 * max(want[m].abs().max().item(), 1.0)
    assert (ln.double() - want)[m].abs().max().item() < tol
    rows = torch.arange(T, device="cuda")[None] < il[:, None]
    assert torch.equal(ref[rows], ref2[rows]) and torch.equal(mp, mp2)


@pytest.mark.parametrize("V", [64, 1024, 8000])
@pytest.mark.parametrize("kind", ["n1", "n2", "peaky", "bias", "offset"])
def test_no_further_from_float64_than_tf32(kind, V):
    """(one to eight parts per tile: the last round's tiles are split along the vocabulary)"""
    E, P, il, ll = make(2, 200, 101, V, std=2.0 if kind == "n2" else 1.0, seed=V)
    g = torch.Generator(device="cuda").manual_seed(1)
    if kind == "peaky":
        E += 6.0 * (torch.rand(E.shape, generator=g, device="cuda") < 0.05)
    if kind == "bias":
        E[:, :, 0] += 4.0
    if kind == "offset":
        E, P = E + 30, P - 30
    m, want = valid(il, ll, 200, 101), truth(E, P)
    rms = {path: (norms(path, E, P, il, ll)[0].double() - want)[m].pow(2).mean().sqrt().item() for path in (2, 4)}
    assert rms[4] <= rms[2]
    a, b = norms(4, E, P, il, ll)[0], norms(4, E, P, il, ll)[0]
    assert torch.equal(a[m], b[m])


@pytest.mark.parametrize("U,gap", [(30, 14.0), (101, 20.0), (150, 45.0), (200, 60.0)])
def test_tiles_beyond_its_range(U, gap):
    """Utterance 1 has one word `gap` above all others in the frames of its second tile and another in every
    position: that tile is the TF32 kernel's bit for bit (its own exact recomputation included), the
    others are not touched.  (A gap near 87 would make the other words' exponentials denormal in the TF32
    kernel's operands, and sums of them lie within the range that it accepts.)"""
    B, T, V = 3, 300, 512
    E, P, _, _ = make(B, T, U, V, seed=U)
    il = torch.tensor([T, T, 200], dtype=torch.int32, device="cuda")
    ll = torch.tensor([U - 1, U - 1, U // 2], dtype=torch.int32, device="cuda")
    P[1, :, 70] += gap
    plain = norms(4, E, P, il, ll)[0]
    E[1, 128:256, 300] += gap
    ln, ref, _ = norms(4, E, P, il, ll)
    tf32 = norms(2, E, P, il, ll)[0]
    m = valid(il, ll, T, U)
    mine = torch.zeros_like(m)
    mine[1, 128:256] = m[1, 128:256]
    assert torch.equal(ln[mine], tf32[mine])
    rest = m & ~mine
    assert torch.equal(ln[rest], plain[rest])
    assert not torch.equal(ln[rest], tf32[rest])
    want = truth(E, P)
    assert (ln.double() - want)[m].abs().max().item() < 8 * 2.0 ** -23 * want[m].abs().max().item() + 4e-6


def test_masked_and_non_finite_words():
    B, T, U, V = 4, 130, 40, 320
    E, P, il, ll = make(B, T, U, V, seed=3)
    il[:], ll[:] = T, U - 1
    lowest = torch.finfo(torch.float32).min
    E[0, :, :200] = float("-inf")     # whole stages masked, the first among them
    E[1, :, 64:128] = lowest
    P[1, :, ::3] = lowest
    E[2, 5, 9] = float("nan")
    E[3, 7, 300] = float("inf")
    ln = norms(4, E, P, il, ll)[0]
    want = truth(E, P)
    fine = torch.isfinite(want)
    assert (ln.double() - want)[fine].abs().max().item() < 2e-5
    assert not torch.isfinite(ln[~fine]).any()


@pytest.mark.parametrize("B,T,U,V", [(2, 200, 40, 1000), (3, 130, 101, 264), (1, 300, 128, 64), (4, 60, 7, 4104)])
def test_bf16_emissions(B, T, U, V):
    """The same numbers in bf16 storage: the same log-normalisers, through the loss (the costs)."""
    E, P, il, ll = make(B, T, U, V, seed=V)
    E, P = E.bfloat16(), P.bfloat16()
    labels = torch.randint(1, V, (B, U - 1), device="cuda", dtype=torch.int32)
    abi.set_option("lognorm_path", 4)
    try:
        a = abi.loss_forward(E, P, labels, il, ll)["costs"]
        b = abi.loss_forward(E.float(), P.float(), labels, il, ll)["costs"]
    finally:
        abi.set_option("lognorm_path", 0)
    assert torch.equal(a, b)


def test_log_norms_that_gradients_may_follow():
    """tb200_log_norms feeds the separate forward and backward calls: on more than 2^24 scores it stays with the
    kernel that the training call takes, bit for bit."""
    E, P, il, ll = make(2, 300, 30, 32000, seed=1)
    assert E.numel() > 1 << 24
    m = valid(il, ll, 300, 30)
    auto, tf32, f16 = (norms(path, E, P, il, ll)[0][m] for path in (0, 2, 4))
    assert torch.equal(auto, tf32) and not torch.equal(auto, f16)
