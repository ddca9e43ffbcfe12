"""GPU tests of the SIMT kernels that serve vocabularies TMA cannot address (not a multiple of 4, or
below 32) against a float64 evaluation: the factored log-normaliser at the edges of its tiles
of 32x32 nodes, its steps of 64 words and the clusters that share a tile, and the gradients at the
edges of their tiles of 64x64 and steps of 32, with labels that share columns."""
import ctypes

import numpy as np
import pytest
import torch

import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def make(B, T, U, V, std=1.0, labels_below=None):
    g = torch.Generator(device="cuda").manual_seed(B * T + U * V)
    E = torch.empty((B, T, V), device="cuda").normal_(0, std, generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(0, std, generator=g)
    labels = torch.randint(1, labels_below or V, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    il = torch.randint(max(1, T // 2), T + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    ll = torch.randint(0, U, (B,), generator=g, device="cuda", dtype=torch.int32)
    il[0], ll[0] = T, U - 1
    return E, P, labels, il, ll


@pytest.mark.parametrize("B,T,U,V", [(1, 1, 1, 2), (2, 31, 33, 29), (1, 33, 31, 63), (3, 64, 32, 65),
                                     (2, 40, 5, 129), (1, 20, 7, 8041), (2, 33, 65, 1025), (16, 200, 40, 257),
                                     (1, 70, 200, 321)])
def test_factored_log_normaliser(B, T, U, V):
    E, P, _, il, ll = make(B, T, U, V, std=2.0)
    ln, ref, mp = abi.log_norms(E, P, il, ll)
    d = E.double(), P.double()
    want = torch.logsumexp(d[0][:, :, None] + d[1][:, None], dim=3)
    m = torch.as_tensor(abi.valid_mask(il.cpu().numpy(), ll.cpu().numpy(), T, U), device="cuda")
    # one rounding of the result, one of the logarithm, 2^-22 of an exponential and the sum's own
    bound = want.abs().max().item() * 2.0 ** -23 + 2.0 ** -20
    assert (ln.double() - want)[m].abs().max().item() < bound
    assert torch.equal(ref[0], E[0].max(dim=1)[0]) and torch.equal(mp[0], P[0].max(dim=1)[0])


def test_factored_sum_out_of_range_is_recomputed():
    E, P, _, il, ll = make(2, 50, 9, 77)
    E[:, 3] -= 1000.0 * (torch.arange(77, device="cuda") != 5)    # E's mass on word 5 ...
    P[:, 4] -= 1000.0 * (torch.arange(77, device="cuda") == 5)    # ... which P excludes
    E[0, 7] = float("-inf")
    ln, _, _ = abi.log_norms(E, P, il, ll)
    want = torch.logsumexp(E.double()[:, :, None] + P.double()[:, None], dim=3)
    m = torch.as_tensor(abi.valid_mask(il.cpu().numpy(), ll.cpu().numpy(), 50, 9), device="cuda")
    ok = m & torch.isfinite(want)
    assert (ln.double() - want)[ok].abs().max().item() < 2e-7 * 1000.0
    assert torch.isneginf(ln[0, 7, :int(ll[0]) + 1]).all()


def _spiked(X, height, g, word=None):
    """One word of every row raised: a word of its own, or the same one throughout."""
    i = torch.randint(0, X.shape[2], X.shape[:2] + (1,), generator=g, device="cuda")
    return X.scatter_add(2, i if word is None else torch.full_like(i, word),
                         torch.full(i.shape, float(height), device="cuda"))


@pytest.mark.parametrize("V", [257, 1025])
@pytest.mark.parametrize("scores", ["plain", "wide", "confident_10", "confident_45", "confident_100", "cancelled_10",
                                    "cancelled_45", "log_softmax"])
def test_factored_is_as_close_to_float64_as_exact(scores, V):
    """Whatever the spread of the scores, the factored kernel may not lose digits against the
    exact one.  rms over 67584 nodes; 1.1: its scatter (below 1 % per 10^4 nodes) and the two
    kernels' different last bits."""
    B, T, U = 8, 256, 33
    g = torch.Generator(device="cuda").manual_seed(V)
    E = torch.empty((B, T, V), device="cuda").normal_(generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(generator=g)
    kind, _, h = scores.partition("_")
    if kind == "wide":
        E, P = 5 * E, 5 * P
    elif kind == "confident":
        E, P = _spiked(E, int(h), g), _spiked(P, int(h), g)
    elif kind == "cancelled":
        E, P = _spiked(E, int(h), g, 3), _spiked(P, -int(h), g, 3)
    elif kind == "log":
        E, P = torch.log_softmax(5 * E, 2), torch.log_softmax(5 * P, 2)
    il = torch.full((B,), T, dtype=torch.int32, device="cuda")
    ll = torch.full((B,), U - 1, dtype=torch.int32, device="cuda")
    want = torch.stack([torch.logsumexp(E[b].double()[:, None] + P[b].double()[None], dim=2) for b in range(B)])
    rms = []
    for path in (0, 1):
        abi.set_option("lognorm_path", path)
        try:
            ln = abi.log_norms(E, P, il, ll)[0]
        finally:
            abi.set_option("lognorm_path", 0)
        rms.append((ln.double() - want).pow(2).mean().sqrt().item())
    assert rms[0] <= 1.1 * rms[1]


@pytest.mark.parametrize("B,T,U,V,below", [(1, 1, 2, 3, None), (2, 63, 64, 65, None), (2, 65, 33, 63, 4),
                                           (1, 64, 65, 129, None), (2, 33, 128, 30, None), (3, 100, 20, 257, 3)])
def test_gradients(B, T, U, V, below):
    E, P, labels, il, ll = make(B, T, U, V, labels_below=below)
    deltas = torch.linspace(0.5, 1.5, B, device="cuda")
    fwd = abi.loss_forward(E, P, labels, il, ll)
    eg, pg = abi.loss_backward(E, P, labels, il, ll, fwd, deltas)
    n = lambda x: x.cpu().numpy()
    ref = O.truth64(n(E), n(P), n(labels), n(il), n(ll))
    s = n(deltas)[:, None, None]
    # alphas are rounded to 2^-15 at most, T + U of them along a path (4 sigma); 1e-5: fp32 sums
    tol = 4.0 * np.sqrt(T + U) * 2.0 ** -15 + 1e-5
    assert abi.rel_to_max(n(eg), ref["egrads"] * s) < tol
    assert abi.rel_to_max(n(pg), ref["pgrads"] * s) < tol


@pytest.fixture
def forced():
    """The factored kernel at any size (small problems go to the exact one by themselves)."""
    abi.set_option("lognorm_path", 3)
    yield
    abi.set_option("lognorm_path", 0)


@pytest.mark.parametrize("B,T,U,V", [(1, 1, 1, 2), (2, 31, 33, 29), (1, 33, 31, 63), (3, 64, 32, 65),
                                     (2, 40, 5, 129), (1, 20, 7, 8041), (2, 33, 65, 1025), (1, 70, 200, 321)])
def test_factored_tile_edges(forced, B, T, U, V):
    test_factored_log_normaliser(B, T, U, V)


def test_factored_sum_out_of_range_is_recomputed_after_the_kernel(forced):
    test_factored_sum_out_of_range_is_recomputed()


@pytest.mark.parametrize("B,T,U,V", [(1, 1, 2, 3), (2, 63, 64, 65), (1, 64, 65, 129), (2, 33, 128, 30), (1, 40, 200, 77)])
def test_factored_gradients(forced, B, T, U, V):
    test_gradients(B, T, U, V, None)


def _kernels(fn):
    """Names of the library's kernels that fn launches."""
    lib = abi.lib
    lib.tb200_profile_enable(1)
    try:
        lib.tb200_profile_reset()
        fn()
        buf = ctypes.create_string_buffer(1 << 14)
        lib.tb200_profile_report(buf, len(buf))
    finally:
        lib.tb200_profile_enable(0)
    return {line.split()[0] for line in buf.value.decode().splitlines()}


@pytest.mark.parametrize("B,T,U,V,kernel", [(8, 400, 1, 1025, "exact"), (8, 400, 4, 1025, "exact"), (64, 1000, 3, 1301, "exact"),
                                            (1, 40, 30, 29, "exact"), (1, 300, 9, 1025, "exact"),
                                            (8, 400, 16, 1025, "factored"), (64, 1000, 8, 1301, "factored"),
                                            (2, 44, 7, 23851, "factored"), (4, 64, 300, 1024, "factored")])
def test_narrow_label_axes_take_the_exact_kernel(B, T, U, V, kernel):
    """A tile of the factored kernel is 32 positions wide: below 4 to 9 of them, and for few nodes,
    the exact kernel's warp per node is the faster one (and both give the same sums)."""
    E, P, labels, il, ll = make(B, T, U, V)
    out = {}
    names = _kernels(lambda: out.update(ln=abi.log_norms(E, P, il, ll)[0]))
    assert "lognorm_" + kernel in names and len({"lognorm_exact", "lognorm_factored"} & names) == 1
    want = torch.logsumexp(E[0].double()[:, None] + P[0].double()[None], dim=2)
    assert (out["ln"][0].double() - want).abs().max().item() < want.abs().max().item() * 2.0 ** -23 + 2.0 ** -20
