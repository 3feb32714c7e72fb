"""Launches that start while the grid before them still runs: whatever follows whatever in a stream -- engine call,
evaluation in one launch or two, leaf list whose length a kernel has just written, buffers that are written over --
gets what it gets with the device idle between calls, eagerly and replayed from a graph."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def encoder(nets):
    from brokefish_b200.nn.cuda_impl import FusedEncoder
    return FusedEncoder(nets["B"], int8=True)


@pytest.mark.parametrize("n", [3, 333, 1000])
def test_a_chain_of_calls_is_the_calls_one_by_one(n, encoder, pos4096):
    """Games played by the network's values: the moves come from the evaluation before, boards and leaf lists are
    written over in place between calls."""
    from brokefish_b200 import env
    legal0 = cu(pos4096["legal"].view(np.int64))

    def play(wait):
        stream = torch.cuda.Stream()
        seen = []
        with torch.cuda.stream(stream):
            pause = (lambda: torch.cuda.synchronize()) if wait else (lambda: None)
            boards, control, rep = (cu(pos4096[k][:n]) for k in ("boards", "control", "rep"))
            mask = legal0[:n].clone()
            ring, length = env.empty_history(n)
            key = env.hash_position(boards, control)
            order = torch.arange(n, dtype=torch.int32, device="cuda")
            count = torch.zeros(1, dtype=torch.int32, device="cuda")
            for ply in range(6):
                policy, promo, value = encoder.forward_full(boards, control, rep, mask)
                pause()
                flat = policy.reshape(n, -1).float()
                best = flat.argmax(dim=1)
                move = torch.where(torch.isfinite(flat.gather(1, best[:, None])[:, 0]), best, torch.full_like(best, -1)).to(torch.int32)
                nb, nc, new_key, irreversible, mask, chk = env.step(boards, control, move, None, with_moves=True, hash=key)
                pause()
                ring, length = env.push_history(ring, length, key, irreversible)
                pause()
                code, result = env.terminal(mask, chk, nc, nb, new_key, ring, length)
                pause()
                boards.copy_(nb)
                control.copy_(nc)
                key = new_key
                count.fill_(0)
                count.add_((code == 0).sum().to(torch.int32))
                order.copy_(torch.argsort((code != 0).to(torch.int8), stable=True))
                prior, label, edges, val = (t.clone() for t in encoder.forward_leaves(boards, control, rep, order, count, mask, 96)[-4:])
                pause()
                live = code == 0
                seen += [policy.clone(), value.clone(), mask, ring, length, code, val[live], edges[live], prior[live], label[live]]
                pause()
        torch.cuda.synchronize()
        return seen

    want = play(wait=True)
    for _ in range(3):
        for a, b in zip(play(wait=False), want):
            assert torch.equal(a, b)
    encoder.check_status()


@pytest.mark.parametrize("n", [2, 200, 333])
def test_a_graph_replays_what_the_calls_do(n, encoder, pos4096):
    from brokefish_b200 import env
    boards, control, rep = (cu(pos4096[k][:n]) for k in ("boards", "control", "rep"))
    legal = cu(pos4096["legal"][:n].view(np.int64))
    order = torch.arange(n, dtype=torch.int32, device="cuda")
    count = torch.tensor([n], dtype=torch.int32, device="cuda")

    def calls():
        out = [t for t in encoder.forward_full(boards, control, rep)]
        mask, chk = env.movegen(boards, control)
        edges = encoder.forward_leaves(boards, control, rep, order, count, mask, 96)
        return [t.clone() for t in out] + [mask, chk] + [t.clone() for t in edges]

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = calls()
    for shift in (0, n, 2 * n):
        for t, k in ((boards, "boards"), (control, "control"), (rep, "rep")):
            t.copy_(cu(pos4096[k][shift:shift + n]))
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in replayed]
        for a, b in zip(got, calls()):
            assert torch.equal(a, b)
    encoder.check_status()


@pytest.mark.parametrize("live", [0, 1, 147, 148, 149, 295, 296, 297, 444, 445, 601])
def test_a_list_of_any_length_is_evaluated_once(live, encoder, pos4096):
    """The launch of two-board tiles and that of one-board tiles each find their part of a list."""
    n = 700
    boards, control, rep = (cu(pos4096[k][:n]) for k in ("boards", "control", "rep"))
    want = [t.clone() for t in encoder.forward_full(boards, control, rep)]
    order = torch.randperm(n, generator=torch.Generator().manual_seed(live)).to(torch.int32).cuda()
    count = torch.tensor([live], dtype=torch.int32, device="cuda")
    encoder.forward_leaves(boards, control, rep, order, torch.zeros_like(count), None, 0)
    out = encoder.forward_leaves(boards, control, rep, order, count, None, 0)
    at = order[:live].long()
    for got, w in zip(out, want):
        assert torch.equal(got[at], w[at])
    encoder.check_status()


ARITHMETICS = {"int8": dict(int8=True), "f16": dict(), "e4m3": dict(fp8=True)}


def back_to_back(rounds, keep_busy, device_idle):
    """What the `rounds` return, each a generator of calls: with the device idle after every call, or with every call
    launched while the ones before it still wait behind a long evaluation."""
    seen = []
    with torch.cuda.stream(torch.cuda.Stream()):
        for calls in rounds:
            keep_busy()
            for out in calls():
                if device_idle:
                    torch.cuda.synchronize()
            seen += [t.clone() for t in out]
    torch.cuda.synchronize()
    return seen


@pytest.mark.parametrize("arithmetic", ARITHMETICS)
@pytest.mark.parametrize("n", [3, 333, 1000])
def test_engine_calls_and_evaluations_directly_after_each_other(n, arithmetic, nets, pos4096):
    """Only the framework's own kernels in between: one launch and two, words made and read, boards stepped and read."""
    from brokefish_b200 import env
    from brokefish_b200.nn.cuda_impl import FusedEncoder
    first, second, busy = (FusedEncoder(nets["B"], **ARITHMETICS[arithmetic]) for _ in range(3))
    every = [cu(pos4096[k]) for k in ("boards", "control", "rep")]
    legal = cu(pos4096["legal"].view(np.int64))
    slot = (legal != 0).int().argmax(dim=1)
    word = legal.gather(1, slot[:, None])
    move = torch.where(word[:, 0] != 0, slot * 64 + ((word >> torch.arange(64, device="cuda")) & 1).argmax(dim=1), -1).int()
    key = env.hash_position(*every[:2])

    def calls(lo):
        boards, control, rep, mv, k = (t[lo:lo + n].clone() for t in (*every, move, key))
        mask, chk = env.movegen(boards, control)
        yield
        policy = first.forward_full(boards, control, rep, mask)
        yield
        nb, nc, nk, irreversible, words, check = env.step(boards, control, mv, None, with_moves=True, hash=k)
        yield
        edges = second.forward_priors(nb, nc, rep, words, 96)
        yield
        again = env.hash_position(nb, nc)
        yield mask, chk, *policy, nb, nc, nk, irreversible, words, check, *edges, again

    rounds = [lambda lo=lo: calls(lo) for lo in (0, n, 2 * n)]
    keep_busy = lambda: busy.forward_full(*every)
    want = back_to_back(rounds, keep_busy, True)
    for _ in range(3):
        for a, b in zip(back_to_back(rounds, keep_busy, False), want):
            assert torch.equal(a, b)
    for e in (first, second, busy):
        e.check_status()


@pytest.mark.parametrize("n", [12289, 20011])
def test_large_launches_of_legal_words_and_what_reads_them(n, encoder, pos4096):
    """Legal words by a thread per board let the next grid start before they are stored."""
    from brokefish_b200 import _native, env
    place = torch.arange(n) % 4096
    every = [cu(pos4096[k])[place.cuda()] for k in ("boards", "control", "rep")]
    gen = torch.Generator().manual_seed(n)
    draw, promo = torch.rand(n, generator=gen).cuda(), torch.randint(0, 4, (n,), generator=gen).to(torch.int8).cuda()
    at = lambda t: ctypes.c_void_p(t.data_ptr())

    def terminal():
        boards, control, rep = (t.clone() for t in every)
        mask, chk = env.movegen(boards, control)
        yield
        yield env.terminal(mask, chk, control, boards)

    def priors():
        boards, control, rep = (t.roll(1, 0) for t in every)
        mask, chk = env.movegen(boards, control)
        yield
        yield encoder.forward_priors(boards, control, rep, mask, 96)

    def random_ply():
        boards, control, rep = (t.roll(2, 0) for t in every)
        move = torch.empty(n, dtype=torch.int32, device="cuda")
        mask, chk = env.movegen(boards, control)
        yield
        _native.check(_native.lib().bf_random_ply(0, at(boards), at(control), at(mask), at(draw), at(promo), n, at(move),
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "bf_random_ply")
        yield boards, control, mask, move

    rounds = [terminal, priors, random_ply]
    keep_busy = lambda: encoder.forward_full(*(t[:4096] for t in every))
    want = back_to_back(rounds, keep_busy, True)
    for _ in range(3):
        for a, b in zip(back_to_back(rounds, keep_busy, False), want):
            assert torch.equal(a, b)
    encoder.check_status()
