"""GPU tests of the single-warp Viterbi sweep (label axes of at most 256 positions) against the CPU path, bit for
bit: every number of positions per lane, more frames than the sweep stages, nodes that the log-normaliser
marked and the re-layout recomputes."""
import numpy as np
import pytest

import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def compare_on_given_norms(E, P, il, ll):
    """tb200_viterbi and the CPU path on the same log-normalisers: nothing but the sweep can differ."""
    B, U = P.shape[:2]
    LN = O.log_norms_torch(E, P)[0].contiguous().numpy()
    want = O.viterbi_abi(E, P, LN, il, ll)
    d = abi.case_to_device(dict(E=E, P=P, labels=np.zeros((B, U - 1), np.int32), in_lens=il, lab_lens=ll))
    got = abi.viterbi(d["E"], d["P"], abi.dev(LN), d["il"], d["ll"]).cpu().numpy()
    for b, n in enumerate(ll):
        assert np.array_equal(got[b, :n], want[b, :n]), b


@pytest.mark.parametrize("U", [1, 2, 17, 32, 40, 65, 97, 130, 161, 193, 225, 256])
@pytest.mark.parametrize("T", [1, 15, 16, 17, 33, 100])
def test_blocks_and_lanes(T, U):
    rng = np.random.default_rng(1000 * T + U)
    B, V = 3, 33
    E = rng.normal(0, 1.5, (B, T, V)).astype(np.float32)
    P = rng.normal(0, 1.5, (B, U, V)).astype(np.float32)
    il = np.array([T, max(1, T // 2), T], np.int32)
    ll = np.array([U - 1, (U - 1) // 2, 0], np.int32)
    compare_on_given_norms(E, P, il, ll)


def test_more_frames_than_are_staged():
    rng = np.random.default_rng(5)
    T, U, V = 60000, 4, 5
    E = rng.normal(0, 1.5, (1, T, V)).astype(np.float32)
    P = rng.normal(0, 1.5, (1, U, V)).astype(np.float32)
    compare_on_given_norms(E, P, np.array([T], np.int32), np.array([U - 1], np.int32))


def test_marked_nodes_are_recomputed():
    """One word of each frame and another of each position 90 above the rest: the factored sum vanishes."""
    rng = np.random.default_rng(6)
    B, T, U, V = 2, 40, 20, 64
    E = rng.normal(0, 1, (B, T, V)).astype(np.float32)
    P = rng.normal(0, 1, (B, U, V)).astype(np.float32)
    E[:, :, 5] += 90
    P[:, :, 9] += 90
    il, ll = np.array([T, T - 3], np.int32), np.array([U - 1, U // 2], np.int32)
    d = abi.case_to_device(dict(E=E, P=P, labels=np.zeros((B, U - 1), np.int32), in_lens=il, lab_lens=ll))
    got = abi.viterbi_decode(d["E"], d["P"], d["il"], d["ll"]).cpu().numpy()
    want = O.viterbi(E, P, il, ll)
    for b, n in enumerate(ll):
        assert np.array_equal(got[b, :n], want[b, :n]), b
