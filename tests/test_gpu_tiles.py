"""The evaluator on one- and two-board tiles: at every size where the tiling changes, a position's
outputs are those it gets in any other batch, in every arithmetic, and those of the four-board kernel,
which carries the dumps and captures; the tiles' products are exact; and the arithmetic helpers the tiles
use instead of divisions equal division on everything they can be given."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ARITHMETICS = {"int8": dict(int8=True), "f16": {}, "e4m3": dict(fp8=True), "ffn": dict(int8=True, int8_scheme="ffn"),
               "ffn+qkv": dict(int8=True, int8_scheme="ffn+qkv")}


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("arithmetic", ARITHMETICS)
def test_every_tiling_gives_a_position_the_same_outputs(arithmetic, nets, pos4096):
    from brokefish_b200.nn.cuda_impl import FusedEncoder
    enc = FusedEncoder(nets["B"], **ARITHMETICS[arithmetic])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    b, c, r = (cu(pos4096[k]) for k in ("boards", "control", "rep"))
    legal = cu(pos4096["legal"].view(np.int64))
    want = [t.clone() for t in enc.forward_full(b, c, r, legal)]
    priors = [t.clone() for t in enc.forward_priors(b, c, r, legal, 96)]
    for n in (1, 2, sms - 1, sms, sms + 1, 2 * sms - 1, 2 * sms, 2 * sms + 1, 3 * sms, 3 * sms + 1, 4 * sms, 4 * sms + 1,
              6 * sms + 1):
        lo = 4096 - n
        part = [t[lo:] for t in (b, c, r, legal)]
        for got, w in zip(enc.forward_full(*part), want):
            assert torch.equal(got, w[lo:]), n
        for got, w in zip(enc.forward_priors(*part, 96), priors):
            assert torch.equal(got, w[lo:]), n
    # one-board tiles off, and up to two rounds of them
    for one in (0, 2):
        enc.set_one_board(one)
        for n in (1, sms + 1, 2 * sms - 1, 2 * sms + 5):
            for got, w in zip(enc.forward_full(*(t[:n] for t in (b, c, r, legal))), want):
                assert torch.equal(got, w[:n]), (one, n)
    enc.check_status()


@pytest.mark.parametrize("arithmetic", ARITHMETICS)
def test_the_instrumented_kernel_gives_the_small_tiles_outputs(arithmetic, nets, pos4096):
    """Stage dumps, operand captures and the phase clock exist in the four-board kernel alone: what they show
    holds for the kernel that evaluates because both give the same bits."""
    from brokefish_b200.nn.cuda_impl import FusedEncoder
    enc = FusedEncoder(nets["B"], **ARITHMETICS[arithmetic])
    n = 301
    args = [cu(pos4096[k][:n]) for k in ("boards", "control", "rep")] + [cu(pos4096["legal"][:n].view(np.int64))]
    want = [t.clone() for t in enc.forward_full(*args)]
    enc.set_profile(True)
    for got, w in zip(enc.forward_full(*args), want):
        assert torch.equal(got, w)
    enc.set_profile(False)
    enc.check_status()


@pytest.mark.parametrize("rows", [32, 64])
@pytest.mark.parametrize("what", ["s8", "u8", "f16", "e4m3", "f16 heads"])
def test_weight_stationary_products(what, rows):
    """Products of one SM, which the self test alone issues -- those of 64 rows lie in tensor memory as the evaluator's
    products of a pair of SMs do (test_gpu_pairs.py) --, against exact host products: bytes over their full range, fp16 and
    e4m3 operands whose sums are all representable."""
    from brokefish_b200 import _native
    from brokefish_b200.nn.pack import sw128_image
    rng = np.random.default_rng(rows)
    n = 128 if what == "f16 heads" else 256
    if what in ("s8", "u8"):
        a = rng.integers(0 if what == "u8" else -128, 256 if what == "u8" else 128, size=(rows, 256))
        w = rng.integers(-128, 128, size=(n, 256))
        a[0, :], w[0, :] = (255 if what == "u8" else -128), -128
        a_bytes, w_bytes = a.astype(np.uint8 if what == "u8" else np.int8).view(np.uint8), w.astype(np.int8).view(np.uint8)
    else:
        a, w = rng.integers(-2, 3, size=(rows, 256)), rng.integers(-2, 3, size=(n, 256))
        if what == "e4m3":
            a_bytes, w_bytes = (torch.from_numpy(m.astype(np.float32)).to(torch.float8_e4m3fn).view(torch.uint8).numpy()
                                for m in (a, w))
        else:
            a_bytes, w_bytes = a.astype(np.float16).view(np.uint8), w.astype(np.float16).view(np.uint8)
    image = np.concatenate([sw128_image(np.ascontiguousarray(w_bytes[:, s:s + 128])) for s in range(0, w_bytes.shape[1], 128)])
    d_a, d_w, d_out = cu(a_bytes), cu(image), torch.zeros(rows, n, dtype=torch.int32, device="cuda")
    mode = 5 + 2 * ["s8", "u8", "f16", "e4m3", "f16 heads"].index(what) + (rows == 64)
    _native.check(_native.lib().bf_selftest_umma(0, mode, *(ctypes.c_void_p(t.data_ptr()) for t in (d_a, d_w, d_out))),
                  "bf_selftest_umma")
    got = d_out.cpu().numpy()
    if what == "e4m3":
        got = got.view(np.float32)
    elif what.startswith("f16"):
        got = np.ascontiguousarray(got.view(np.float16)[:, ::2])
    assert np.array_equal(got.astype(np.int64), a.astype(np.int64) @ w.astype(np.int64).T)


def test_scales_and_reciprocals_equal_division():
    from brokefish_b200 import _native
    differ = (ctypes.c_ulonglong * 4)()
    _native.check(_native.lib().bf_selftest_scales(0, differ), "bf_selftest_scales")
    assert list(differ) == [0, 0, 0, 0]


@pytest.mark.parametrize("n_value", [1, 3])
@pytest.mark.parametrize("head", ["king", "pooled", "prenorm"])
@pytest.mark.parametrize("arithmetic", ["int8", "f16"])
def test_a_value_does_not_depend_on_the_tile(arithmetic, head, n_value, pos4096):
    """Every value head on one-, two- and four-board tiles, to the bit: fp16 batches change kernels with
    their size, the int8 ones under the phase clock."""
    from brokefish_b200.nn.cuda_impl import FusedEncoder
    from brokefish_b200.nn.model import net_for_state, seeded_state
    state = seeded_state(seed=11, std=None, perturb_norms=True, n_value=n_value, value_head=head)
    net = net_for_state(state).eval()
    net.load_state_dict(state)
    enc = FusedEncoder(net, **ARITHMETICS[arithmetic])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    b, c, r = (cu(pos4096[k]) for k in ("boards", "control", "rep"))
    legal = cu(pos4096["legal"].view(np.int64))
    want = [t.clone() for t in enc.forward_full(b, c, r)]
    assert float(want[2].abs().max()) > 0.05
    for n in (1, sms, sms + 1, 2 * sms + 1, 4 * sms, 4 * sms + 1):
        for got, w in zip(enc.forward_full(b[:n], c[:n], r[:n]), want):
            assert torch.equal(got, w[:n]), n
    # the expansion's warps share a buffer with the prenorm head
    n = 2 * sms + 5
    assert torch.equal(enc.forward_priors(b[:n], c[:n], r[:n], legal[:n], 96)[3], want[2][:n])
    enc.set_profile(True)
    for got, w in zip(enc.forward_full(b[:n], c[:n], r[:n]), want):
        assert torch.equal(got, w[:n])
    enc.set_profile(False)
    enc.check_status()
    enc.close()
