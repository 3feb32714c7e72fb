"""The work a program has this framework do, as cases that can be timed and compared.

Six uses, each through the public entry points:

* ``evaluate``: positions to logits and values (``FusedEncoder.forward_full``), from the one
  position of an analysis board over a search's batches to a self-play or training batch; in
  the shipped int8 arithmetic, in the default fp16 and in the e4m3 one; raw or with the
  legality words ANDed into the policy;
* ``expand``: positions straight to the edges and priors of their search nodes
  (``forward_priors``), the legal moves given or generated in the kernel;
* ``leaves``: the live part of a search's staged leaves, its length known to the device only
  (``forward_leaves``);
* ``host``: the end-to-end call on pinned host buffers (``forward_host`` for logits,
  ``forward_priors_host`` for edge lists);
* ``ply``: one ply of many games at once: the move, the new legal moves and key, the repetition
  ring and the game-end rules (``step``, ``push_history``, ``terminal``);
* ``movegen``: legal moves of positions that are already there (``movegen``).

Positions are uniform-random games of up to 120 plies from the start position, played on the
device; networks have the shipped shape with seeded random weights, biases and norms.
"""

import math
import random

import torch

from brokefish_b200 import env
from brokefish_b200.nn.cuda_impl import FusedEncoder
from brokefish_b200.nn.model import BrokefishNet

ARITHMETICS = {"int8": dict(int8=True), "f16": dict(), "e4m3": dict(fp8=True)}
#: Bytes of the packed weights, read once per pass.
WEIGHT_BYTES = {"int8": 6_475_000, "f16": 12_770_000, "e4m3": 8_575_000}
#: 32 weight GEMMs, the attention products and the head product of one position.
FLOPS = 402_653_184 + 8_388_608 + 32 * 256 * 71 * 2
#: boards, control word, repetition count; policy, promotion logits, value.
BYTES_IN, BYTES_OUT = 67, 4356
#: Games that are played to make positions; larger batches draw from them.
MOST_GAMES = 16384


def listed():
    return [
        # an analysis board or a game against a human: one position at a time, latency is all
        {"name": "evaluate-1", "use": "evaluate", "arithmetic": "int8", "n": 1, "masked": False},
        # one search tree's batch of leaves
        {"name": "evaluate-64", "use": "evaluate", "arithmetic": "int8", "n": 64, "masked": True},
        # a few trees searched together: neither a power of two nor a multiple of anything
        {"name": "evaluate-333", "use": "evaluate", "arithmetic": "int8", "n": 333, "masked": False},
        # the self-play leaf batch, the size that the framework is quoted at
        {"name": "evaluate-4096", "use": "evaluate", "arithmetic": "int8", "n": 4096, "masked": False},
        # the constructor's default arithmetic at a search batch
        {"name": "evaluate-f16-1000", "use": "evaluate", "arithmetic": "f16", "n": 1000, "masked": False},
        # the e4m3 arithmetic at its configured batch, a training-data labelling pass
        {"name": "evaluate-e4m3-16384", "use": "evaluate", "arithmetic": "e4m3", "n": 16384, "masked": False},
        # search nodes from positions, moves generated in the kernel
        {"name": "expand-777", "use": "expand", "n": 777, "e_cap": 96, "given": False},
        # a search with early termination: a seventh of its staged leaves is live
        {"name": "leaves-600-of-4096", "use": "leaves", "staged": 4096, "live": 600, "e_cap": 96},
        # an engine in another process or language: host buffers in, logits out
        {"name": "host-4096", "use": "host", "n": 4096, "priors": False},
        # the same for search nodes of a smaller tree
        {"name": "host-priors-100", "use": "host", "n": 100, "priors": True},
        # self-play: one ply of every game
        {"name": "ply-4096", "use": "ply", "n": 4096},
        # legality words for a data set
        {"name": "movegen-1048576", "use": "movegen", "n": 1048576},
    ]


def _spread(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    use = rng.choices(["evaluate", "expand", "leaves", "host", "ply", "movegen"], [8, 2, 2, 3, 3, 2])[0]
    if use == "evaluate":
        arithmetic = rng.choices(["int8", "f16", "e4m3"], [4, 1, 1])[0]
        return {"use": use, "arithmetic": arithmetic, "n": _spread(rng, 1, 15000), "masked": rng.random() < 0.3}
    if use == "expand":
        return {"use": use, "n": _spread(rng, 1, 8192), "e_cap": rng.choice([64, 96, 128]),
                "given": rng.random() < 0.5}
    if use == "leaves":
        staged = _spread(rng, 64, 8192)
        return {"use": use, "staged": staged, "live": _spread(rng, 1, staged), "e_cap": rng.choice([0, 96])}
    if use == "host":
        return {"use": use, "n": _spread(rng, 1, 8192), "priors": rng.random() < 0.5}
    if use == "ply":
        return {"use": use, "n": _spread(rng, 1, 131072)}
    return {"use": use, "n": _spread(rng, 1, 1048576)}


def _positions(n: int, seed: int):
    """``n`` positions with their legality words: boards, control, repetition counts, legal."""
    games = min(n, MOST_GAMES)
    boards, control, rep, legal, _ = env.random_playouts(games, seed)
    if games == n:
        return boards, control, rep, legal
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pick = torch.randint(0, games, (n,), generator=gen, device="cuda")
    return boards[pick], control[pick], rep[pick], legal[pick]


def _encoder(arithmetic: str, seed: int) -> FusedEncoder:
    """An evaluator of a network with weights, biases and norms drawn from the seed."""
    gen = torch.Generator().manual_seed(seed)
    net = BrokefishNet().eval()
    with torch.no_grad():
        for name, p in net.named_parameters():
            if p.dim() >= 2:
                std = p.shape[1] ** -0.5
                p.copy_(torch.randn(p.shape, generator=gen) * std)
            else:
                gamma = "norm" in name and name.endswith("weight")
                p.copy_(0.1 * torch.randn(p.shape, generator=gen) + (1.0 if gamma else 0.0))
    return FusedEncoder(net, **ARITHMETICS[arithmetic])


def _moves(legal: torch.Tensor, seed: int) -> torch.Tensor:
    """One legal move per board, the lowest target square of a random slot that can move; -1 without a move."""
    gen = torch.Generator(device=legal.device).manual_seed(seed + 1)
    can = legal != 0
    slot = (torch.rand(legal.shape, generator=gen, device=legal.device) + can).argmax(dim=1)
    word = legal.gather(1, slot[:, None]).squeeze(1)
    bits = (word[:, None] >> torch.arange(64, device=legal.device)) & 1
    move = slot * 64 + bits.argmax(dim=1)
    return torch.where(can.any(dim=1), move, torch.full_like(move, -1)).to(torch.int32)


def prepare(case, seed):
    use = case["use"]
    state = {"use": use}
    n = case["staged"] if use == "leaves" else case["n"]
    boards, control, rep, legal = _positions(n, seed)
    if use == "movegen":
        return {**state, "args": (boards, control)}
    if use == "ply":
        gen = torch.Generator(device="cuda").manual_seed(seed + 2)
        key = env.hash_position(boards, control)
        ring, length = env.empty_history(n)
        # games in progress: up to forty plies since the last irreversible move, some of which
        # have been at this position before
        length.copy_(torch.randint(0, 41, (n,), generator=gen, device="cuda"))
        ring.copy_(torch.randint(-2 ** 62, 2 ** 62, ring.shape, generator=gen, device="cuda"))
        again = torch.rand(ring.shape, generator=gen, device="cuda") < 0.02
        ring = torch.where(again, key[:, None], ring)
        promo = torch.randint(0, 4, (n,), generator=gen, device="cuda").to(torch.int8)
        return {**state, "args": (boards, control, _moves(legal, seed), promo, key, ring, length)}
    state["encoder"] = encoder = _encoder(case.get("arithmetic", "int8"), seed)
    if use == "evaluate":
        return {**state, "args": (boards, control, rep, legal if case["masked"] else None)}
    if use == "expand":
        return {**state, "args": (boards, control, rep, legal if case["given"] else None, case["e_cap"])}
    if use == "leaves":
        # every place has been evaluated once before, as in a search that is under way
        order = torch.randperm(n, generator=torch.Generator().manual_seed(seed)).to(torch.int32).cuda()
        count = torch.tensor([n], dtype=torch.int32, device="cuda")
        e_cap = case["e_cap"]
        encoder.forward_leaves(boards, control, rep, order, count, legal if e_cap else None, e_cap)
        live = torch.tensor([case["live"]], dtype=torch.int32, device="cuda")
        return {**state, "args": (boards, control, rep, order, live, legal if e_cap else None, e_cap)}
    pinned = [t.cpu().pin_memory() for t in (boards, control, rep, legal)]
    if case["priors"]:
        out = [torch.empty(n, 96, dtype=torch.half), torch.empty(n, 96, dtype=torch.int16),
               torch.empty(n, dtype=torch.int32), torch.empty(n)]
        state["call"], ins = encoder.forward_priors_host, pinned
    else:
        out = [torch.empty(n, 32, 64, dtype=torch.half), torch.empty(n, 32, 4, dtype=torch.half), torch.empty(n)]
        state["call"], ins = encoder.forward_host, pinned[:3]
    return {**state, "args": (*ins, *(t.pin_memory() for t in out))}


def run(state):
    use, args = state["use"], state["args"]
    if use == "evaluate":
        return state["encoder"].forward_full(*args)
    if use == "expand":
        return state["encoder"].forward_priors(*args)
    if use == "leaves":
        return state["encoder"].forward_leaves(*args)
    if use == "host":
        return state["call"](*args)
    if use == "movegen":
        return env.movegen(*args)
    boards, control, move, promo, key, ring, length = args
    boards, control, new_key, irreversible, mask, in_check = env.step(boards, control, move, promo,
                                                                      with_moves=True, hash=key)
    ring, length = env.push_history(ring, length, key, irreversible)
    code, result = env.terminal(mask, in_check, control, boards, new_key, ring, length)
    return boards, control, new_key, irreversible, mask, in_check, ring, length, code, result


def work(case):
    use = case["use"]
    if use == "movegen":                   # board and control word in, legal words and check flag out
        return {"bytes": case["n"] * (66 + 257), "flops": 0}
    if use == "ply":
        # board, control, move, promotion, key, ring, length in; board, control, key, flags, legal
        # words, ring, length, code and result out
        return {"bytes": case["n"] * (66 + 4 + 1 + 8 + 808 + 66 + 8 + 2 + 256 + 808 + 2), "flops": 0}
    weights = WEIGHT_BYTES[case.get("arithmetic", "int8")]
    if use == "evaluate":
        return {"bytes": weights + case["n"] * (BYTES_IN + BYTES_OUT + (256 if case["masked"] else 0)),
                "flops": case["n"] * FLOPS}
    if use == "expand":
        return {"bytes": weights + case["n"] * (BYTES_IN + 4 * case["e_cap"] + 8 + (256 if case["given"] else 0)),
                "flops": case["n"] * FLOPS}
    if use == "leaves":
        out = BYTES_OUT + 256 + 4 * case["e_cap"] + 4 if case["e_cap"] else BYTES_OUT
        return {"bytes": weights + case["live"] * (4 + BYTES_IN + out), "flops": case["live"] * FLOPS}
    out = 256 + 4 * 96 + 8 if case["priors"] else BYTES_OUT
    return {"bytes": weights + case["n"] * (BYTES_IN + out), "flops": case["n"] * FLOPS}


def tolerance(case):
    if case["use"] in ("ply", "movegen"):
        return "exact"
    # fp16 logits of an eight-layer network on 8-bit or fp16 operands: one rounding that falls the
    # other way early on moves an operand by a step; with a cut edge list a near tie may change
    # which edges stay
    return {"rel": 1e-2, "max": 0.1, "differ": 1e-3}
