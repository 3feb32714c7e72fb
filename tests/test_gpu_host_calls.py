"""The host-buffer calls (C ABI bf_forward_host, bf_forward_priors_host) give the device call's bits
whatever buffers they are given and whichever way that takes them."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def enc(nets):
    from brokefish_b200.nn.cuda_impl import FusedEncoder
    e = FusedEncoder(nets["B"], int8=True)
    yield e
    e.check_status()
    e.close()


class Buffer:
    """Host memory of a call: `array` as bytes (or as many zero bytes), `offset` bytes into an allocation."""

    def __init__(self, array=None, nbytes=0, pinned=True, offset=0):
        raw = None if array is None else np.ascontiguousarray(array).view(np.uint8).reshape(-1)
        size = nbytes if raw is None else raw.size
        whole = torch.zeros(size + 64, dtype=torch.uint8)
        if pinned:
            whole = whole.pin_memory()
        self.bytes = whole[offset:offset + size]
        if raw is not None:
            self.bytes.copy_(torch.from_numpy(raw))
        self.ptr = ctypes.c_void_p(self.bytes.data_ptr())

    def same(self, tensor):
        return np.array_equal(self.bytes.numpy(), tensor.cpu().contiguous().numpy().view(np.uint8).reshape(-1))


def inputs(pos, n, **kw):
    return [Buffer(pos[k][:n], **kw) for k in ("boards", "control", "rep", "legal")]


def device_inputs(pos, n):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a[:n])).cuda()
    return t(pos["boards"]), t(pos["control"]), t(pos["rep"]), t(pos["legal"].view(np.int64))


def logits_call(enc, n, ins, outs, legal=True):
    from brokefish_b200 import _native
    b, c, r, lg = (x.ptr for x in ins)
    _native.check(_native.lib().bf_forward_host(enc._handle, b, c, r, lg if legal else None, n,
                                                *(x.ptr if x else None for x in outs)), "bf_forward_host")


def edges_call(enc, n, e_cap, ins, outs):
    from brokefish_b200 import _native
    _native.check(_native.lib().bf_forward_priors_host(enc._handle, *(x.ptr for x in ins), n, e_cap,
                                                       *(x.ptr if x else None for x in outs)), "bf_forward_priors_host")


def logits_buffers(n, **kw):
    return [Buffer(nbytes=n * k, **kw) for k in (4096, 256, 4)]


def edges_buffers(n, e_cap, **kw):
    return [Buffer(nbytes=n * k, **kw) for k in (2 * e_cap, 2 * e_cap, 4, 4)]


@pytest.mark.parametrize("n,plan", [(1, 0), (64, 0), (2500, 2)])
@pytest.mark.parametrize("offset", [2, 4, 8])
def test_pinned_buffers_may_start_anywhere(offset, n, plan, enc, pos4096):
    """Off the boundaries that the kernels' 16- and 8-byte accesses need: in the small call, which would
    otherwise work in the buffers themselves, and in the plan whose last launch writes into them."""
    want = [t.clone() for t in enc.forward_full(*device_inputs(pos4096, n))]
    edges = [t.clone() for t in enc.forward_priors(*device_inputs(pos4096, n), 96)]
    enc.set_host_plan(plan)
    moved, straight = inputs(pos4096, n, offset=offset), inputs(pos4096, n)
    for ins, off in ((moved, offset), (moved, 0), (straight, offset)):
        outs = logits_buffers(n, offset=off)
        logits_call(enc, n, ins, outs)
        assert all(o.same(w) for o, w in zip(outs, want)), (ins is moved, off)
        outs = edges_buffers(n, 96, offset=off)
        edges_call(enc, n, 96, ins, outs)
        assert all(o.same(w) for o, w in zip(outs, edges)), (ins is moved, off)
    enc.set_host_plan(0)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 2500])
def test_logits_on_every_way(n, enc, pos4096):
    """Work in the caller's buffers (all pinned, up to 64 positions) and the copies (more, or any buffer
    pageable), with and without legality words, every output or some."""
    b, c, r, lg = device_inputs(pos4096, n)
    want = {True: [t.clone() for t in enc.forward_full(b, c, r, lg)]}
    want[False] = [t.clone() for t in enc.forward_full(b, c, r)]
    for legal in (True, False):
        ways = [[True] * 7, [False] * 7] + [[i != k for i in range(7)] for k in range(7)]
        for pinned in ways:
            ins = [Buffer(pos4096[k][:n], pinned=p) for k, p in zip(("boards", "control", "rep", "legal"), pinned)]
            outs = [Buffer(nbytes=n * k, pinned=p) for k, p in zip((4096, 256, 4), pinned[4:])]
            logits_call(enc, n, ins, outs, legal)
            assert all(o.same(w) for o, w in zip(outs, want[legal])), (legal, pinned)
        for keep in range(1, 7):
            outs = [o if keep >> i & 1 else None for i, o in enumerate(logits_buffers(n))]
            logits_call(enc, n, inputs(pos4096, n), outs, legal)
            assert all(o.same(w) for o, w in zip(outs, want[legal]) if o), (legal, keep)


@pytest.mark.parametrize("waves", ["one", "last in place", "first copied", "several"])
def test_edge_lists_on_every_way(waves, enc, pos4096):
    """The same for edge lists, which are written in place up to four positions per SM; an edge cap that is
    no multiple of eight has its rows off the 16-byte boundaries."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = {"one": 1, "last in place": 4 * sms, "first copied": 4 * sms + 1, "several": 2500}[waves]
    for e_cap in (96, 13):
        want = [t.clone() for t in enc.forward_priors(*device_inputs(pos4096, n), e_cap)]
        ways = [[True] * 8, [False] * 8] + [[i != k for i in range(8)] for k in range(8)]
        for pinned in ways:
            ins = [Buffer(pos4096[k][:n], pinned=p) for k, p in zip(("boards", "control", "rep", "legal"), pinned)]
            outs = [Buffer(nbytes=n * k, pinned=p) for k, p in zip((2 * e_cap, 2 * e_cap, 4, 4), pinned[4:])]
            edges_call(enc, n, e_cap, ins, outs)
            assert all(o.same(w) for o, w in zip(outs, want)), (e_cap, pinned)
        for pinned in (True, False):
            outs = edges_buffers(n, e_cap, pinned=pinned)[:3] + [None]       # no values wanted
            edges_call(enc, n, e_cap, inputs(pos4096, n, pinned=pinned), outs)
            assert all(o.same(w) for o, w in zip(outs[:3], want)), (e_cap, pinned)
