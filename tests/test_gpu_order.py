"""Launches that start while the grid before them still runs: whatever follows whatever in a stream -- engine call,
evaluation in one launch or two, leaf list whose length a kernel has just written, buffers that are written over --
gets what it gets with the device idle between calls, eagerly and replayed from a graph."""
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
                seen += [policy.clone(), value.clone(), mask, ring, length, code, val[live], edges[live]]
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
