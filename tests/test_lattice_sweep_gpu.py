"""GPU tests of the lattice sweeps (label axes of at most 256 positions) against a float64
evaluation at the edges of what they are cut into: blocks of 16 diagonals, the positions a lane
owns (1, 2, 4, 5..8), tiles of 32 frames, empty and one-node lattices.  The exact SIMT kernels stand
around the sweeps, so that what is compared is theirs."""
import threading

import numpy as np
import pytest
import torch

import abi
from oracle import oracle as O
from transducer_b200 import TransducerLoss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,U", [(1, 1), (1, 2), (15, 1), (16, 1), (17, 16), (16, 17), (31, 2), (32, 33),
                                 (33, 32), (64, 64), (47, 65), (130, 127), (128, 128), (5, 128), (400, 40),
                                 (1, 129), (50, 160), (33, 161), (70, 192), (16, 193), (40, 225), (100, 256)])
def test_edges(T, U):
    B, V = 4, 40
    g = torch.Generator(device="cuda").manual_seed(100 * T + U)
    E = torch.empty((B, T, V), device="cuda").normal_(generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(generator=g)
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.randint(max(1, T // 2), T + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    ll = torch.randint(0, U, (B,), generator=g, device="cuda", dtype=torch.int32)
    il[0], ll[0], il[3] = T, U - 1, 0
    abi.set_option("lognorm_path", 1)
    abi.set_option("grads_path", 1)
    try:
        fwd = abi.loss_forward(E, P, labels, il, ll)
        eg, pg = abi.loss_backward(E, P, labels, il, ll, fwd)
        eg2, pg2 = abi.loss_backward(E, P, labels, il, ll, fwd)   # the saved state is not consumed
        torch.cuda.synchronize()
    finally:
        abi.set_option("lognorm_path", 0)
        abi.set_option("grads_path", 0)
    assert torch.equal(eg, eg2) and torch.equal(pg, pg2)
    n = lambda x: x.cpu().numpy()
    ref = O.truth64(n(E), n(P), n(labels), n(il), n(ll))
    # A stored alpha is below 1024 in magnitude for these scores (up to 128 positions: at most two blocks
    # of 16 arcs of up to 20 below its block's offset; beyond: at T + U <= 356) and rounded to 2^-14,
    # 2^-15 at most, which is what the T + U factors of a path carry, independently: 4 sigma.
    # 1e-5: the fp32 contractions.
    tol = 4.0 * np.sqrt(T + U) * 2.0 ** -15 + 1e-5
    costs = n(fwd["costs"])
    np.testing.assert_allclose(costs[:3], ref["costs"][:3], rtol=1e-6, atol=tol)
    assert np.isposinf(costs[3])
    assert abi.rel_to_max(n(eg), ref["egrads"]) < tol
    assert abi.rel_to_max(n(pg), ref["pgrads"]) < tol


def costs_alone(E, P, labels, il, ll):
    """Costs [B] and their sum by the call that no backward call follows."""
    lib, (B, T, V), U = abi.lib, E.shape, P.shape[1]
    costs, total = torch.zeros((B,), device="cuda"), torch.zeros((1,), device="cuda")
    n = lib.tb200_loss_score_workspace_bytes(B, T, U, V)
    ws = abi.workspace(n)
    abi.use_torch_stream()
    abi.check(lib.tb200_loss_score(*[abi.ptr(t) for t in (E, P, labels, il, ll, costs, total)], B, T, U, V, 0,
                                   abi.ptr(ws), n))
    return costs, total


@pytest.mark.parametrize("S", [1, 2, 15, 16, 17, 30, 31, 32, 33, 47, 48, 49, 63, 64, 65, 96])
def test_around_the_middle_diagonal(S):
    """Costs alone: the halves of an utterance meet at a multiple of 16 diagonals.  Lattices of S diagonals,
    short and long label axes (every number of positions per lane), utterances whose middle lies
    elsewhere beside them."""
    for U in (1, 2, 9, 33, 40, 65, 129, 161, 193, 225):
        T = S + 1 - U
        if T < 1:
            T, U = S // 3 + 1, S - S // 3   # (the axes swapped: more positions than frames)
        B, V = 3, 36
        g = torch.Generator(device="cuda").manual_seed(1000 * S + U)
        E = torch.empty((B, T, V), device="cuda").normal_(generator=g)
        P = torch.empty((B, U, V), device="cuda").normal_(generator=g)
        labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
        il = torch.tensor([T, max(1, T // 2), T], dtype=torch.int32, device="cuda")
        ll = torch.tensor([U - 1, U - 1, (U - 1) // 2], dtype=torch.int32, device="cuda")
        abi.set_option("lognorm_path", 1)
        try:
            costs, total = costs_alone(E, P, labels, il, ll)
        finally:
            abi.set_option("lognorm_path", 0)
        n = lambda x: x.cpu().numpy()
        ref = O.truth64(n(E), n(P), n(labels), n(il), n(ll))
        tol = 4.0 * np.sqrt(T + U) * 2.0 ** -15 + 1e-5   # (as test_edges)
        np.testing.assert_allclose(n(costs), ref["costs"], rtol=1e-6, atol=tol)
        np.testing.assert_allclose(total.item(), ref["costs"].sum(), rtol=1e-6, atol=3 * tol)


@pytest.mark.parametrize("U", [5, 40, 100, 150])
def test_an_utterance_without_a_path(U):
    """Costs alone, every label of utterance 1 masked by -inf: its cost is +inf, and the others do not notice."""
    B, T, V = 3, 50, 40
    g = torch.Generator(device="cuda").manual_seed(U)
    E = torch.empty((B, T, V), device="cuda").normal_(generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(generator=g)
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.full((B,), T, dtype=torch.int32, device="cuda")
    ll = torch.full((B,), U - 1, dtype=torch.int32, device="cuda")
    whole, _ = costs_alone(E, P, labels, il, ll)
    E[1, :, 1:] = float("-inf")
    costs, _ = costs_alone(E, P, labels, il, ll)
    assert torch.isposinf(costs[1])
    assert torch.equal(costs[[0, 2]], whole[[0, 2]])


def test_host_threads_with_different_shapes():
    """Stream and error message are per host thread, a kernel's shared-memory limit is not: a thread's
    launches may not depend on what another one set for a shorter utterance.  (200 positions: the
    sweep that stages T blank emissions.)"""
    def worker(T, failures):
        with torch.cuda.stream(torch.cuda.Stream()):
            E, P = torch.randn((1, T, 32), device="cuda"), torch.randn((1, 200, 32), device="cuda")
            labels = torch.ones((1, 199), dtype=torch.int32, device="cuda")
            il = torch.tensor([T], dtype=torch.int32, device="cuda")
            ll = torch.tensor([199], dtype=torch.int32, device="cuda")
            for _ in range(400):
                try:
                    fwd = abi.loss_forward(E, P, labels, il, ll)
                    abi.loss_backward(E, P, labels, il, ll, fwd)
                except Exception as e:
                    failures.append((T, str(e)))
            torch.cuda.current_stream().synchronize()

    failures = []
    threads = [threading.Thread(target=worker, args=(T, failures)) for T in (8, 3000, 16, 2000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]


@pytest.mark.parametrize("T,U,std,bias,masked", [(130, 100, 15.0, 0.0, False), (200, 30, 3.0, 25.0, False),
                                                 (90, 160, 15.0, 0.0, False), (60, 60, 1.0, 0.0, True),
                                                 (60, 170, 1.0, 0.0, True)])
def test_large_and_masked_scores(T, U, std, bias, masked):
    """Arcs far larger than N(0,1) scores give, and words masked by -inf (from the second frame on, so
    that every node stays reachable).  How large a stored alpha gets depends on the arcs, and
    so does what its rounding costs."""
    B, V, blank = 3, 40, 0
    g = torch.Generator(device="cuda").manual_seed(T * U)
    E = torch.empty((B, T, V), device="cuda").normal_(0, std, generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(0, std, generator=g)
    E[:, :, blank] += bias
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.tensor([T, T - 1, T // 2], dtype=torch.int32, device="cuda")
    ll = torch.tensor([U - 1, U // 2, U - 2], dtype=torch.int32, device="cuda")
    E_ref = E.clone()
    if masked:
        hide = torch.rand((B, T - 1, V - 1), generator=g, device="cuda") < 0.2
        E[:, 1:, 1:].masked_fill_(hide, float("-inf"))
        E_ref[:, 1:, 1:].masked_fill_(hide, -1e4)   # (the oracle's lattice wants finite scores)
    abi.set_option("lognorm_path", 1)
    abi.set_option("grads_path", 1)
    try:
        fwd = abi.loss_forward(E, P, labels, il, ll)
        eg, pg = abi.loss_backward(E, P, labels, il, ll, fwd)
    finally:
        abi.set_option("lognorm_path", 0)
        abi.set_option("grads_path", 0)
    n = lambda x: x.cpu().numpy()
    ref = O.truth64(n(E_ref), n(P), n(labels), n(il), n(ll))
    # largest arc a path takes, in nats: among the best of each node, as an upper bound the blank's
    lse = torch.logsumexp(E.double()[:, :, None] + P.double()[:, None], dim=3)
    arc = (lse - E[:, :, None, blank] - P[:, None, :, blank]).max().item()
    # a stored alpha: up to 128 positions at most 32 arcs below its offset, in log2 units; beyond, the
    # whole path.  Rounded to half an ulp, T + U of them along a path, independently: 4 sigma, and
    # twice that for the three roundings of an arc's sum.
    size = 32 * arc * 1.4427 if U <= 128 else float(np.max(ref["costs"])) + 32 * arc
    tol = 8.0 * np.sqrt(T + U) * 2.0 ** -25 * size + 1e-5
    assert tol < 0.05
    np.testing.assert_allclose(n(fwd["costs"]), ref["costs"], rtol=1e-6, atol=tol)
    assert abi.rel_to_max(n(eg), ref["egrads"]) < tol
    assert abi.rel_to_max(n(pg), ref["pgrads"]) < tol


@pytest.mark.parametrize("T,U", [(1, 129), (60, 150), (31, 161), (90, 200), (40, 225), (100, 256), (4200, 256)])
def test_wide_axes_against_the_row_major_kernel(T, U):
    """Axes of 129..256 positions (natural logarithms at full magnitude) against the kernel behind
    tb200_forward on the same log-normalisers; more frames than the sweep stages (4096 at 256
    positions) included."""
    B, V = 3, 36
    g = torch.Generator(device="cuda").manual_seed(T + U)
    E = torch.empty((B, T, V), device="cuda").normal_(0, 3, generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(0, 3, generator=g)
    E[1, :, 1:].masked_fill_(torch.rand((T, V - 1), generator=g, device="cuda") < 0.2, float("-inf"))
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.tensor([T, T, max(1, T // 2)], dtype=torch.int32, device="cuda")
    ll = torch.tensor([U - 1, U - 2, U // 2], dtype=torch.int32, device="cuda")
    abi.set_option("lognorm_path", 1)
    try:
        ln = abi.log_norms(E, P, il, ll)[0]
        costs = abi.loss_forward(E, P, labels, il, ll)["costs"]
    finally:
        abi.set_option("lognorm_path", 0)
    want = abi.forward(E, P, ln, labels, il, ll)[0]
    # per node of a path of T + U: 2^-22 of the hardware logaddexp, three roundings of an alpha (4 sigma)
    finite = torch.isfinite(want)
    tol = (T + U) * 2.0 ** -22 + 4.0 * (3 * (T + U)) ** 0.5 * 2.0 ** -24 * want[finite].max().item()
    assert finite[0] and finite[2]   # (the masked utterance of one frame has no path)
    assert (costs - want)[finite].abs().max().item() < tol and torch.equal(costs[~finite], want[~finite])


@pytest.mark.parametrize("T,U", [(1, 1), (40, 9), (33, 65), (100, 128), (1, 129), (60, 150), (33, 161), (90, 200),
                                 (40, 225), (700, 256), (20, 257)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_costs_alone(T, U, dtype):
    """The call without a backward call to follow against float64, through the module as well (which takes it
    under no_grad and where no input requires a gradient); beyond 128 positions it has sweeps of its own."""
    B, V = 3, 40
    if dtype == "bf16" and U > 128:
        pytest.skip("bf16: label axes of at most 128 positions")
    g = torch.Generator(device="cuda").manual_seed(10 * T + U)
    E = torch.empty((B, T, V), device="cuda").normal_(generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(generator=g)
    if dtype == "bf16":
        E, P = E.bfloat16(), P.bfloat16()
    labels = torch.randint(1, V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.tensor([T, max(1, T // 2), 0], dtype=torch.int32, device="cuda")
    ll = torch.tensor([U - 1, U // 2 if U > 1 else 0, U - 1], dtype=torch.int32, device="cuda")
    lib = abi.lib
    costs, total = torch.zeros((B,), device="cuda"), torch.zeros((1,), device="cuda")
    n = lib.tb200_loss_score_workspace_bytes(B, T, U, V)
    ws = abi.workspace(n)
    abi.use_torch_stream()
    fn = lib.tb200_loss_score_bf16 if dtype == "bf16" else lib.tb200_loss_score
    args = [abi.ptr(t) for t in (E, P, labels, il, ll, costs, total)] + [B, T, U, V, 0, abi.ptr(ws)]
    assert fn(*args, n - 256) == 1   # (too small a workspace is refused)
    abi.check(fn(*args, n))
    h = lambda x: x.float().cpu().numpy()
    ref = O.truth64(h(E), h(P), labels.cpu().numpy(), il.cpu().numpy(), ll.cpu().numpy())["costs"]
    # as test_edges, and 2^-19 a node for the log-normalisers (tensor cores)
    tol = 4.0 * np.sqrt(T + U) * 2.0 ** -15 + 1e-5 + (T + U) * 2.0 ** -19
    np.testing.assert_allclose(h(costs)[:2], ref[:2], rtol=1e-6, atol=tol)
    assert np.isposinf(h(costs)[2])
    crit = TransducerLoss()
    with torch.no_grad():
        quiet = crit(E, P, labels, il, ll)
    plain = crit(E, P, labels, il, ll)
    E.requires_grad_(True)
    graded = crit(E, P, labels, il, ll)
    assert torch.equal(quiet, costs) and torch.equal(plain, costs) and not quiet.requires_grad
    assert graded.requires_grad
    # with gradients to follow, axes beyond 128 positions carry alphas at full magnitude: three roundings of
    # them a node (4 sigma), and 2^-22 of the hardware logaddexp
    if U > 128:
        tol += (T + U) * 2.0 ** -22 + 4.0 * (3 * (T + U)) ** 0.5 * 2.0 ** -24 * float(np.max(ref[:2]))
    np.testing.assert_allclose(h(graded.detach())[:2], h(costs)[:2], rtol=1e-6, atol=2 * tol)
