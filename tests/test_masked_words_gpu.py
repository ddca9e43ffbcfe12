"""Words masked by -inf or by a very low number, through the costs with gradients and the costs alone: the same answers,
against float64."""
import numpy as np
import pytest
import torch

from transducer_b200 import TransducerLoss

pytestmark = pytest.mark.gpu

INF, LOWEST = float("inf"), torch.finfo(torch.float32).min


def truth(E, P, labels, il, ll, blank=0):
    """Costs in float64, +inf where there is no path."""
    out = []
    for b in range(E.shape[0]):
        T, U = int(il[b]), int(ll[b]) + 1
        e, p = E[b, :T].double().cpu(), P[b, :U].double().cpu()
        ln = torch.stack([torch.logsumexp(e[t][None] + p, 1) for t in range(T)]).numpy()
        stay = (e[:, None, blank] + p[None, :, blank]).numpy() - ln
        lab = labels[b, :U - 1].long().cpu()
        step = (e[:, lab] + p[torch.arange(U - 1), lab][None]).numpy() - ln[:, :U - 1]
        a = np.full((T, U), -np.inf)
        a[0, 0] = 0.0
        for t in range(T):
            for u in range(U):
                if t:
                    a[t, u] = np.logaddexp(a[t, u], a[t - 1, u] + stay[t - 1, u])
                if u:
                    a[t, u] = np.logaddexp(a[t, u], a[t, u - 1] + step[t, u - 1])
        out.append(-(a[T - 1, U - 1] + stay[T - 1, U - 1]))
    return np.array(out)


def case(U, mask):
    """Utterance 0 has a label that can never be emitted: no path.  1: nothing masked.  2: position 2 cannot stay
    and its word is masked in frame 4, a node that nothing leads to although paths exist.  3: half of the words
    masked in a stretch of frames, and the blank in one of the positions."""
    g = torch.Generator(device="cuda").manual_seed(U)
    B, T, V = 4, 60, 64
    E = torch.empty((B, T, V), device="cuda").normal_(0, 1, generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(0, 1, generator=g)
    labels = torch.randint(6, V, (B, U - 1), device="cuda", generator=g, dtype=torch.int32)
    il = torch.tensor([T, T, T - 9, T], device="cuda", dtype=torch.int32)
    ll = torch.tensor([U - 1, U - 1, U // 2, U - 1], device="cuda", dtype=torch.int32)
    labels[0, 3] = 1
    P[0, 3, 1] = mask
    labels[2, :3] = 5
    P[2, 2, 0] = mask
    E[2, 4, 5] = mask
    E[3, 10:20, 1:33] = mask
    P[3, 4, 0] = mask
    return E, P, labels, il, ll


@pytest.mark.parametrize("U", [8, 20, 40, 70, 100, 128, 151, 200])
@pytest.mark.parametrize("mask", [-INF, LOWEST, -1e30, -1e4])
def test_costs_with_and_without_gradients(U, mask):
    E, P, labels, il, ll = case(U, mask)
    want = truth(E, P, labels, il, ll)
    loss = TransducerLoss()
    with torch.no_grad():
        alone = loss(E, P, labels, il, ll).cpu().double().numpy()
    E.requires_grad_(), P.requires_grad_()
    costs = loss(E, P, labels, il, ll)
    with_grads = costs.detach().cpu().double().numpy()
    costs[1:].sum().backward()
    if mask < -1e29:
        # a cost beyond 3.8e29 is no path to the costs alone, and to both up to 128 positions
        assert alone[0] == INF and (with_grads[0] == INF if U <= 128 or mask == -INF else with_grads[0] > 9e29)
    for got in (alone, with_grads):
        first = 1 if mask < -1e29 else 0
        np.testing.assert_allclose(got[first:], want[first:], rtol=1e-5)
    for b in (1, 2, 3):
        assert torch.isfinite(E.grad[b]).all() and torch.isfinite(P.grad[b]).all()


@pytest.mark.parametrize("U", [20, 100, 151])
@pytest.mark.parametrize("mask", [-1e20, -1e29])
def test_forced_paths_through_very_low_scores(U, mask):
    """A path of huge but finite cost is a path."""
    E, P, labels, il, ll = case(U, mask)
    loss = TransducerLoss()
    with torch.no_grad():
        alone = loss(E, P, labels, il, ll)
    with_grads = loss(E.requires_grad_(), P, labels, il, ll).detach()
    for got in (alone, with_grads):
        assert abs(got[0].item() / -mask - 1.0) < 1e-5


@pytest.mark.parametrize("U", [20, 70, 151, 250])
def test_gradients_beside_nodes_that_nothing_leads_to(U):
    """A mask of -1e4 has the same gradients as -inf to the last bit that a float64 sum could show: there every number is
    ordinary."""
    grads = []
    for mask in (-INF, -1e4):
        E, P, labels, il, ll = case(U, mask)
        E.requires_grad_(), P.requires_grad_()
        TransducerLoss()(E, P, labels, il, ll)[1:].sum().backward()
        grads.append((E.grad[1:], P.grad[1:]))
    for a, b in zip(*grads):
        # (the log-normalisers of both are computed alike; 1e-5: the sums of a few hundred fp32 occupancies)
        assert (a - b).abs().max().item() <= 1e-5 * max(b.abs().max().item(), 1.0)
