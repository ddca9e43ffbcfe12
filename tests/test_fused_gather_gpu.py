"""GPU tests of the two ways in which the label and blank emissions reach the lattice: handed out by the
tensor-core log-normaliser (large inputs) or gathered by the re-layout (inputs that stay in
L2).  Both are the same numbers, so costs and gradients are compared bit for bit, at the edges of
the hand-out: odd T, tails of the vocabulary, blank last, repeated labels, every width of the
label axis, bf16 storage."""
import pytest
import torch

import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,U,V,blank,dtype,below", [
    (2, 131, 33, 128, 0, "f32", None), (1, 257, 2, 36, 35, "f32", None), (3, 77, 101, 260, 259, "f32", 5),
    (2, 301, 128, 1000, 7, "f32", None), (2, 140, 1, 64, 0, "f32", None),
    (2, 259, 129, 132, 131, "f32", None), (2, 150, 151, 512, 0, "f32", 4), (1, 385, 201, 1000, 3, "f32", None),
    (2, 133, 256, 264, 263, "f32", None),
    (2, 131, 33, 128, 0, "bf16", None), (3, 77, 101, 264, 263, "bf16", 5), (1, 129, 2, 32, 0, "bf16", None),
    (2, 301, 128, 1000, 7, "bf16", None)])
def test_hand_out_and_gather_agree(B, T, U, V, blank, dtype, below):
    g = torch.Generator(device="cuda").manual_seed(B * T + U + V)
    E = torch.empty((B, T, V), device="cuda").normal_(generator=g)
    P = torch.empty((B, U, V), device="cuda").normal_(generator=g)
    if dtype == "bf16":
        E, P = E.bfloat16(), P.bfloat16()
    labels = torch.randint(0, below or V - 1, (B, U - 1), generator=g, device="cuda", dtype=torch.int32)
    labels[labels >= blank] += 1
    il = torch.randint(max(1, T // 2), T + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    ll = torch.randint(0, U, (B,), generator=g, device="cuda", dtype=torch.int32)
    il[0], ll[0] = T, U - 1
    out = []
    for mode in (0, 2, 1):
        abi.set_option("fused_gather", mode)
        try:
            fwd = abi.loss_forward(E, P, labels, il, ll, blank=blank)
            out.append((fwd["costs"],) + abi.loss_backward(E, P, labels, il, ll, fwd, blank=blank))
        finally:
            abi.set_option("fused_gather", 1)
    abi.check(abi.lib.tb200_check_status())
    assert torch.isfinite(out[0][0]).all()
    for other in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(out[0], other))
