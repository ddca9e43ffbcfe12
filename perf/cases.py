"""The work a user of transducer_b200 has it do, as cases that can be timed and compared.

Every case goes through `TransducerLoss`: training steps (loss and both gradients), scoring
(loss only, no gradient) and teacher-forced Viterbi decoding.  Shapes, length ranges and value
distributions are those of `transducer_b200/workloads.py` and the tests, plus generic ones in
between.  A case is a dict:

    task      "train" (costs, d/d emissions, d/d predictions of the mean cost), "score" (costs
              under no_grad) or "viterbi" (labels of the best alignment)
    B T U V   utterances, frames, longest transcript (predictions have U + 1 rows), vocabulary
    t_min u_min  lengths are uniform in [t_min, T] and [u_min, U]; utterance 0 is full length
    std peak blank_bias  scores are N(0, std); a share `peak` of the emissions is raised by 6; the
              blank column of the emissions is raised by blank_bias
    last_blank   the blank is the last word of the vocabulary instead of word 0
    dtype     "f32" or "bf16" storage of emissions, predictions and their gradients
    checked   the constructor's defaults (lengths validated, device status read back: the call
              synchronises) or validate_lengths=False (the call only enqueues work)
"""
import math

import torch

from transducer_b200 import TransducerLoss


def _case(name, task, B, T, U, V, t_min=None, u_min=None, std=1.0, peak=0.0, blank_bias=0.0,
          last_blank=False, dtype="f32", checked=False):
    case = {"task": task, "B": B, "T": T, "U": U, "V": V,
            "t_min": T if t_min is None else t_min, "u_min": U if u_min is None else u_min,
            "std": std, "peak": peak, "blank_bias": blank_bias, "last_blank": last_blank,
            "dtype": dtype, "checked": checked}
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest call: two short utterances over a character set (launches and host work count)
        _case("train_tiny_v30", "train", 2, 50, 10, 30, t_min=25, u_min=1, checked=True),
        # characters on long, unsubsampled utterances, all of full length: the lattice dominates
        _case("train_v100", "train", 8, 2000, 100, 100, checked=True),
        # a small word-piece vocabulary on the same utterances
        _case("train_v1000", "train", 8, 2000, 100, 1000),
        # 1024 word pieces and a blank behind them, ragged mid-sized utterances: rows of an odd length
        _case("train_v1025_odd", "train", 16, 600, 80, 1025, t_min=250, u_min=20, last_blank=True,
              checked=True),
        # a large vocabulary on a small batch of long utterances
        _case("train_v10000_b8", "train", 8, 2000, 100, 10000),
        # the large batch the headline is quoted on
        _case("train_v10000_b32", "train", 32, 2000, 100, 10000, t_min=1500, u_min=60, std=2.0),
        # the same from a mixed-precision model: bf16 scores in, bf16 gradients out
        _case("train_v10000_b32_bf16", "train", 32, 2000, 100, 10000, t_min=1500, u_min=60, std=2.0,
              dtype="bf16"),
        # long transcripts: a label axis of more than 128 positions
        _case("train_u150_v4096", "train", 64, 1500, 150, 4096, t_min=750, u_min=75, blank_bias=4.0),
        # scoring one short utterance (a hypothesis re-scored while a user waits)
        _case("score_one_v512", "score", 1, 400, 40, 512, checked=True),
        # scoring with a large word-piece vocabulary and peaky emissions: one GPU's 64 of 256 utterances
        _case("score_v32000", "score", 64, 1000, 200, 32000, t_min=500, u_min=100, peak=0.05),
        # best alignment of a small batch over a small vocabulary
        _case("viterbi_v500", "viterbi", 8, 400, 60, 500, t_min=200, u_min=20, blank_bias=4.0,
              checked=True),
        # best alignment of a large batch of long utterances
        _case("viterbi_v4096", "viterbi", 64, 1500, 150, 4096, t_min=750, u_min=75, blank_bias=4.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges: 1-64 utterances, 40-2000 frames, transcripts of 4-200 labels,
    28-32000 words (half of the vocabularies a multiple of 8, as models are padded to; the others
    as they come, and those that are not a multiple of 4 on at most 1e8 scores)."""
    while True:
        task = rng.choice(["train", "train", "train", "score", "viterbi", "viterbi"])
        B, T, V = _log(rng, 1, 64), _log(rng, 40, 2000), _log(rng, 28, 32000)
        U = _log(rng, 4, min(200, T // 2))
        if rng.random() < 0.5:
            V = (V + 7) // 8 * 8
        bf16 = task != "viterbi" and V % 8 == 0 and V >= 32 and U <= 127 and rng.random() < 0.4
        ragged = rng.random() < 0.7
        case = _case(None, task, B, T, U, V,
                     t_min=max(1, int(T * rng.uniform(0.4, 0.9))) if ragged else T,
                     u_min=max(1, int(U * rng.uniform(0.2, 0.9))) if ragged else U,
                     std=rng.choice([1.0, 1.0, 2.0]), peak=rng.choice([0.0, 0.0, 0.05]),
                     blank_bias=4.0 if task == "viterbi" or rng.random() < 0.3 else 0.0,
                     last_blank=rng.random() < 0.3, dtype="bf16" if bf16 else "f32",
                     checked=rng.random() < 0.5)
        scores = B * T * V
        if scores > (2e9 if task == "score" else 6.4e8) or (V % 4 and scores > 1e8):
            continue
        # per lattice node the decoding's comparisons cost more than the other tasks' products
        if task == "viterbi" and scores * U > 64 * 1500 * 150 * 4096 * 0.75:
            continue
        return case


def prepare(case, seed):
    dev = torch.device("cuda")
    B, T, U, V = case["B"], case["T"], case["U"], case["V"]
    blank = V - 1 if case["last_blank"] else 0
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    E = torch.empty((B, T, V), device=dev).normal_(0.0, case["std"], generator=g)
    P = torch.empty((B, U + 1, V), device=dev).normal_(0.0, case["std"], generator=g)
    if case["peak"]:
        for b in range(B):
            E[b] += 6.0 * (torch.rand((T, V), generator=g, device=dev) < case["peak"])
    if case["blank_bias"]:
        E[:, :, blank] += case["blank_bias"]
    if case["dtype"] == "bf16":
        E, P = E.bfloat16(), P.bfloat16()
    first = 0 if case["last_blank"] else 1   # the labels are the words other than the blank
    labels = torch.randint(first, first + V - 1, (B, U), generator=g, device=dev, dtype=torch.int32)
    in_lens = torch.randint(case["t_min"], T + 1, (B,), generator=g, device=dev, dtype=torch.int32)
    lab_lens = torch.randint(case["u_min"], U + 1, (B,), generator=g, device=dev, dtype=torch.int32)
    in_lens[0], lab_lens[0] = T, U
    if case["task"] == "train":
        E.requires_grad_(True)
        P.requires_grad_(True)
    criterion = TransducerLoss(blank=blank) if case["checked"] \
        else TransducerLoss(blank=blank, validate_lengths=False)
    # (entries of a decoded row beyond its utterance's length are unspecified)
    padding = torch.arange(U, device=dev)[None, :] >= lab_lens[:, None]
    return {"task": case["task"], "criterion": criterion, "E": E, "P": P, "labels": labels,
            "in_lens": in_lens, "lab_lens": lab_lens, "padding": padding}


def run(state):
    criterion, E, P = state["criterion"], state["E"], state["P"]
    if state["task"] == "viterbi":
        best = criterion.viterbi(E, P, state["in_lens"], state["lab_lens"])
        return best.masked_fill_(state["padding"], 0)
    if state["task"] == "score":
        with torch.no_grad():
            return criterion(E, P, state["labels"], state["in_lens"], state["lab_lens"])
    costs = criterion(E, P, state["labels"], state["in_lens"], state["lab_lens"])
    dE, dP = torch.autograd.grad(costs.mean(), (E, P))
    return {"costs": costs.detach(), "dE": dE, "dP": dP}


def _lengths(case):
    """Expected sums over the batch: frames, label positions, lattice nodes."""
    B = case["B"]
    t, u = (case["t_min"] + case["T"]) / 2, (case["u_min"] + case["U"]) / 2 + 1
    return (case["T"] + (B - 1) * t, case["U"] + 1 + (B - 1) * u,
            case["T"] * (case["U"] + 1) + (B - 1) * t * u)


def work(case):
    """Inputs read once (valid rows), outputs written once (gradients whole, padding included); the
    products of the log-normaliser and of both gradients, for Viterbi the log-normaliser's products
    and one addition and one comparison per node and word."""
    frames, positions, nodes = _lengths(case)
    B, T, U, V = case["B"], case["T"], case["U"], case["V"]
    size = 2 if case["dtype"] == "bf16" else 4
    out = 4.0 * B
    if case["task"] == "train":
        out += size * V * B * (T + U + 1.0)
    elif case["task"] == "viterbi":
        out = 4.0 * B * U
    flops = {"train": 6.0, "score": 2.0, "viterbi": 4.0}[case["task"]] * V * nodes
    return {"bytes": size * V * (frames + positions) + 4.0 * B * (U + 2) + out, "flops": flops}


def tolerance(case):
    """About four times the largest distance seen between the tensor-core path and the exact fp32
    path, or the same path with more operand splits, over these cases and drawn ones: costs 1e-6
    (32-bit sums over up to 2000 frames: 1e-5 stated), fp32 gradients 1.3e-4 (weights of the two
    contractions rounded to TF32) with single entries up to 1.8e-3, bf16 gradients 5e-4 with single
    entries up to 1e-2 (a neighbouring bf16 number).  Decoded labels agreed throughout; a path may
    turn where two of its scores round to a tie."""
    if case["task"] == "viterbi":
        return {"rel": 1e-5, "differ": 1e-3}
    if case["task"] == "score":
        return {"rel": 1e-5}
    return {"rel": 2e-3, "max": 0.04} if case["dtype"] == "bf16" else {"rel": 5e-4, "max": 7e-3}
