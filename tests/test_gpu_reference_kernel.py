"""The product against the reference's OWN kernel, both on the same GPU.

``oracle/build_ref.py`` compiles the reference's ``csrc/encoder.cu`` for sm_100a from the
reference checkout and saves the weight slabs the reference's constructor derives; this file
runs that kernel (``oracle/ref_kernel.py``) and the product on identical seeded positions and
weights.  The built reference is not part of the history: on a machine with a GPU these tests fail
without it, after all others have run.

Bar for the int8 arithmetic (the path the metric is quoted on): BIT IDENTITY.  The product
keeps the reference kernel's own rounding points and summation orders -- LayerNorm partial
sums and butterfly, hardware 1/sqrt, fp16 accumulation in the attention products
(``mma.sync``) and in the head product (tcgen05 with fp16 accumulators, which gives the same
bits), ``__expf`` softmax, the fused multiply-add in the ff2 running total -- and runs the
exact-integer GEMMs on tcgen05, so every layer-0 debug stage, the final norm after
eight layers, policy, promo and value come out equal to the bit (measured on 2048 positions
for four weight sets: 0 differing elements, value difference 0.0, argmax agreement 100 %).

The e4m3-FFN arithmetic is a tolerance: there the product accumulates its fp16 and e4m3
tcgen05 GEMMs in fp32 where the reference accumulates in fp16 (measured 6.3 % of max|logit|;
the reference's own bar for a quantised path is 8 % of max|logit| against fp32).
"""
import os

import numpy as np
import pytest
import torch

from conftest import GOLDEN

from oracle import int8_encoder as O
from oracle import ref_kernel as R

pytestmark = [pytest.mark.gpu]


@pytest.fixture(autouse=True)
def _checker_is_built():
    """On a box with a GPU a missing checker is a failure, not a skip: these tests are the
    bit-identity evidence, and a silent skip would drop it."""
    assert R.available(), ("oracle/_ref is not built: run `python -c 'import __graft_entry__ as g; "
                           "g.build()'` where the reference's sources are at hand")

SETS = {"A": dict(seed=0, std=0.02, perturb_norms=False),
        "B": dict(seed=0, std=None, perturb_norms=True)}


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def inputs(pos, sl):
    return dev(pos["boards"][sl]), dev(pos["control"][sl]), dev(pos["rep"][sl])


def product(state_kw, **enc_kw):
    from brokefish_b200.nn import encoder_impl
    from brokefish_b200.nn.model import net_for_state, seeded_state
    st = seeded_state(**state_kw)
    net = net_for_state(st).eval()
    net.load_state_dict(st)
    if "fp8" not in enc_kw:
        enc_kw.setdefault("int8", True)      # the shipped arithmetic unless a test asks otherwise
    return encoder_impl("cuda")(net, **enc_kw)


def run_both(enc, ref, pos, sl):
    mine = [t.cpu().numpy().copy() for t in enc.forward_full(*inputs(pos, sl))]
    enc.check_status()
    theirs = [t.cpu().numpy().copy() for t in ref.forward_full(*inputs(pos, sl))]
    torch.cuda.synchronize()
    return mine, theirs


def rel_tol(theirs_pol, frac):
    return frac * max(1.0, float(np.abs(theirs_pol.astype(np.float32)).max()))


def check_argmax(pol, rpol, legal, floor, tol):
    mine, theirs = O.masked_argmax(pol, legal), O.masked_argmax(rpol, legal)
    playable = theirs >= 0
    assert (mine[playable] == theirs[playable]).mean() >= floor
    flat = rpol.astype(np.float32).reshape(rpol.shape[0], -1)
    for i in np.where(playable & (mine != theirs))[0]:
        assert flat[i, theirs[i]] - flat[i, mine[i]] <= tol


def same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("name", ["A", "B"])
def test_int8_outputs_are_bit_identical_to_the_reference_kernel(name, pos256):
    if not R.available(f"{name}_int8"):
        pytest.skip("slabs missing")
    enc, ref = product(SETS[name]), R.RefKernel(f"{name}_int8")
    assert (ref.quant, ref.two_boards) == (3, 1) and not enc.exact_rsqrt
    sl = slice(0, 256)
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, sl)
    assert same_bits(pol, rpol) and same_bits(pro, rpro)
    assert np.abs(val - rval).max() <= 1e-6
    # an odd batch, so the reference's spare board slot and the product's partial tile are hit
    odd = slice(5, 5 + 77)
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, odd)
    assert same_bits(pol, rpol) and same_bits(pro, rpro) and np.abs(val - rval).max() <= 1e-6
    enc.close()


@pytest.mark.parametrize("name", ["A", "B"])
def test_every_debug_stage_is_bit_identical(name, pos256):
    """Stage 9 embedding; layer 0: 1 LN1, 5/6/7 Q/K/V, 4 attention output, 2 residual after
    attention, 3 LN2; 8 the final norm after all eight layers (the reference's stage numbers,
    csrc/encoder.cu:1315-1596)."""
    if not R.available(f"{name}_int8"):
        pytest.skip("slabs missing")
    enc, ref = product(SETS[name]), R.RefKernel(f"{name}_int8")
    sl = slice(0, 200)
    for stage in (9, 1, 5, 6, 7, 4, 2, 3, 8):
        got = enc.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        want = ref.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        assert same_bits(got, want), stage
    enc.close()


def test_int8_full_batch_is_bit_identical(pos4096):
    if not R.available("A_int8"):
        pytest.skip("slabs missing")
    enc, ref = product(SETS["A"]), R.RefKernel("A_int8")
    sl = slice(0, 4096)
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos4096, sl)
    assert same_bits(pol, rpol) and same_bits(pro, rpro)
    assert np.abs(val - rval).max() <= 1e-6
    mine, theirs = O.masked_argmax(pol, pos4096["legal"][sl]), O.masked_argmax(rpol, pos4096["legal"][sl])
    assert np.array_equal(mine, theirs)
    enc.close()


def test_every_batch_size_of_the_sweep_is_bit_identical():
    """Batch sizes 1 .. 65536 of the batch-sweep configuration (piece counts uniform in 2..32 by
    extra captures, side to move flipped on half the boards, seed 2), with the sizes around a
    tile (4 boards) and around one wave (148 CTAs x 4 boards) added: ragged last tiles, CTAs
    without work, and many waves all give the reference kernel's bits."""
    if not R.available("B_int8"):
        pytest.skip("slabs missing")
    from brokefish_b200.positions import varied
    enc, ref = product(SETS["B"]), R.RefKernel("B_int8")
    b, c, r, _ = varied(65536, seed=2)
    pieces = ((b.view(np.uint16) >> 11) & 1) == 0
    assert pieces.sum(1).min() == 2 and pieces.sum(1).max() == 32 and 0.4 < (c < 0).mean() < 0.6
    for n in (1, 2, 3, 4, 5, 63, 64, 65, 511, 512, 513, 591, 592, 593, 4096, 16384, 65536):
        lo = 0 if n == 65536 else 65536 - n - 7
        args = [dev(a[lo:lo + n]) for a in (b, c, r)]
        pol, pro, val = [t.cpu().numpy().copy() for t in enc.forward_full(*args)]
        rpol, rpro, rval = [t.cpu().numpy().copy() for t in ref.forward_full(*args)]
        assert same_bits(pol, rpol) and same_bits(pro, rpro), n
        assert np.abs(val - rval).max() <= 1e-6, n
    enc.check_status()
    enc.close()


def test_reinjection_is_bit_identical(pos256):
    if not R.available("C_int8_rj"):
        pytest.skip("slabs missing")
    kw = dict(seed=7, std=None, perturb_norms=True, reinject="both")
    enc, ref = product(kw), R.RefKernel("C_int8_rj")
    assert ref.rj_mode == 2 and enc.rj_mode == 2
    sl = slice(0, 96)
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, sl)
    assert same_bits(pol, rpol) and same_bits(pro, rpro) and np.abs(val - rval).max() <= 1e-6
    enc.close()


@pytest.mark.parametrize("name,kw,mode", [
    ("C_f16_rj", dict(seed=7, std=None, perturb_norms=True, reinject="both"), 2),
    ("D_f16_rj1", dict(seed=8, std=0.02, perturb_norms=True, reinject="ln1"), 1)])
def test_reinjection_on_the_fp16_arithmetic_is_bit_identical(name, kw, mode, pos256):
    """The reference builds re-injection for its int8 and its fp16 kernel
    (brokefish/nn/cuda_impl.py:413-420); so does this library, both modes."""
    if not R.available(name):
        pytest.skip("slabs missing")
    enc, ref = product(kw, int8=False), R.RefKernel(name)
    assert ref.rj_mode == mode and enc.rj_mode == mode and ref.quant == 0 and enc.quant == 0
    sl = slice(0, 96)
    for stage in (1, 3, 8):
        got = enc.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        want = ref.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        assert same_bits(got, want), stage
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, sl)
    assert same_bits(pol, rpol) and same_bits(pro, rpro) and np.abs(val - rval).max() <= 1e-6
    enc.close()
    with pytest.raises(NotImplementedError):
        product(kw, fp8=True)


def test_pooled_wdl_value_is_bit_identical(pos256):
    if not R.available("V_int8_wdl"):
        pytest.skip("slabs missing")
    kw = dict(seed=3, std=0.02, perturb_norms=True, n_value=3, value_head="pooled")
    enc, ref = product(kw), R.RefKernel("V_int8_wdl")
    assert (ref.n_value, ref.vmode) == (3, 1)
    sl = slice(0, 96)
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, sl)
    assert same_bits(pol, rpol) and same_bits(pro, rpro) and np.abs(val - rval).max() <= 1e-6
    enc.close()


def test_prenorm_wdl_value_against_reference_kernel(pos256):
    """The prenorm value head pools the raw residual and norms it once; the product sums in
    another order than the reference's one warp (csrc/encoder.cu:1008-1057), all in fp32, so the
    value is held to 1e-5 while policy and promo stay bit-identical."""
    if not R.available("P_int8_prenorm"):
        pytest.skip("slabs missing")
    kw = dict(seed=5, std=None, perturb_norms=True, n_value=3, value_head="prenorm")
    enc, ref = product(kw), R.RefKernel("P_int8_prenorm")
    assert (ref.n_value, ref.vmode) == (3, 2)
    sl = slice(0, 96)
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, sl)
    assert same_bits(pol, rpol) and same_bits(pro, rpro)
    assert np.abs(val - rval).max() <= 1e-5
    enc.close()


#: What the e4m3 arm is held to against the reference's e4m3 kernel, per weight set:
#: max |dlogit| as a fraction of max |logit| -- the reference's own bar for a quantised path,
#: 8 % (tests/test_quant.py:342-356) -- and the masked-argmax agreement at 16384 positions
#: (measured value minus a small margin; set A's N(0, 0.02) weights give nearly flat logits, so
#: its argmax is decided by differences far below the tolerance; set B has default-init scale).
#: Measured on a B200: set A 6.2 % / 6.5 % of max|logit| (256 / 16384 positions), value 0.047,
#: agreement 0.9496, worst regret 0.067; set B 4.7 %, value 0.102, agreement 0.9578, regret 0.083.
E4M3_BARS = {"A": dict(rel=8e-2, value=8e-2, agree=0.94), "B": dict(rel=8e-2, value=1.2e-1, agree=0.95)}


@pytest.mark.parametrize("name", ["A", "B"])
def test_e4m3_arm_against_the_reference_e4m3_kernel(name, pos256):
    """The e4m3-FFN arithmetic.  Its fp16 GEMMs (QKV, out-projection) run on tcgen05 with fp16
    accumulators, which carry the bits of the reference's fp16-accumulate mma.sync, so layer 0 is
    bit-identical up to the FFN input: LN1, Q, K, V, attention output, residual, LN2.  The FFN
    itself accumulates e4m3 products in fp32 where the reference accumulates in fp16 (no tcgen05
    form reproduces that instruction's roundings), so the outputs are a tolerance, the reference's
    own for a quantised path: 8 % of max|logit|."""
    assert R.available(f"{name}_e4m3"), "slabs missing: rebuild oracle/_ref"
    bars = E4M3_BARS[name]
    enc, ref = product(SETS[name], fp8=True), R.RefKernel(f"{name}_e4m3")
    assert ref.quant == 1
    sl = slice(0, 128)
    for stage in (9, 1, 5, 6, 7, 4, 2, 3):
        got = enc.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        want = ref.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        assert same_bits(got, want), stage
    (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos256, sl)
    d = np.abs(pol.astype(np.float32) - rpol.astype(np.float32)).max()
    top = np.abs(rpol.astype(np.float32)).max()
    print(f"e4m3 arm, set {name}, vs reference e4m3 kernel: max|dlogit| {d:.4f} = {d / top:.4f} of max|logit| "
          f"{top:.3f}, value {np.abs(val - rval).max():.4f}")
    assert d <= rel_tol(rpol, bars["rel"])
    assert np.abs(val - rval).max() <= bars["value"]
    # the 16384-position configuration (piece counts 2..32, side to move flipped on half, seed 3):
    # same tolerance, everything finite, and the masked argmax of the two kernels agrees on
    # most positions that have a legal move
    from brokefish_b200.positions import varied
    b, c, r, lg = varied(16384, seed=3)
    args = [dev(a) for a in (b, c, r)]
    pol, pro, val = [t.cpu().numpy().copy() for t in enc.forward_full(*args)]
    rpol, rpro, rval = [t.cpu().numpy().copy() for t in ref.forward_full(*args)]
    enc.check_status()
    assert np.isfinite(pol.astype(np.float32)).all() and np.isfinite(val).all()
    d = np.abs(pol.astype(np.float32) - rpol.astype(np.float32)).max()
    top = np.abs(rpol.astype(np.float32)).max()
    dv = float(np.abs(val - rval).max())
    alive = ((b.view(np.uint16) >> 11) & 1) == 0
    lg = np.where(alive, lg, 0)                       # captured pieces have no moves
    has_move = lg.any(axis=1) & (c > 0)               # words are the mover's only where nothing was flipped
    mine, theirs = O.masked_argmax(pol, lg), O.masked_argmax(rpol, lg)
    agree = (mine == theirs)[has_move].mean()
    # how much worse than the reference kernel's choice the product's choice is, by the
    # reference kernel's own logits
    flat = rpol.astype(np.float32).reshape(rpol.shape[0], -1)
    rows = np.where(has_move & (mine != theirs))[0]
    regret = float((flat[rows, theirs[rows]] - flat[rows, mine[rows]]).max()) if rows.size else 0.0
    print(f"e4m3, set {name}, 16384 positions: max|dlogit| {d:.4f} = {d / top:.4f} of max|logit| {top:.3f}, "
          f"value {dv:.4f}, masked-argmax agreement {agree:.4f} on {has_move.sum()}, worst regret {regret:.4f}")
    assert d <= rel_tol(rpol, bars["rel"]) and dv <= bars["value"]
    assert agree >= bars["agree"]
    assert regret <= rel_tol(rpol, bars["rel"])
    enc.close()


@pytest.mark.parametrize("name", ["A", "V_int8_wdl"])
def test_small_batches_in_the_one_board_form_keep_the_bits(name, pos256):
    """A batch of at most one board per SM runs in the small-batch form of the kernel (one board
    per tile, replicated in the four lane quadrants, sixteen row warps per board).  Its policy,
    promotion logits and values equal the four-board form's and the reference kernel's bit for
    bit, for the king-row scalar head and for the pooled win/draw/loss head, at one position, at
    odd counts and at the largest count that still takes the form; the fused expansion and the
    leaf list go through it too."""
    kw = SETS["A"] if name == "A" else dict(seed=3, std=0.02, perturb_norms=True, n_value=3, value_head="pooled")
    ref_name = "A_int8" if name == "A" else name
    assert R.available(ref_name)
    enc, ref = product(kw), R.RefKernel(ref_name)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (1, 3, 37, sms - 1, sms):
        sl = slice(11, 11 + n)
        enc.set_one_board(1)
        mine = [t.clone() for t in enc.forward_full(*inputs(pos256, sl))]
        enc.check_status()
        enc.set_one_board(0)
        four = [t.clone() for t in enc.forward_full(*inputs(pos256, sl))]
        theirs = [t.clone() for t in ref.forward_full(*inputs(pos256, sl))]
        torch.cuda.synchronize()
        for a, b, c in zip(mine, four, theirs):
            assert same_bits(a.cpu().numpy(), b.cpu().numpy()), n
        assert same_bits(mine[0].cpu().numpy(), theirs[0].cpu().numpy()) and same_bits(mine[1].cpu().numpy(), theirs[1].cpu().numpy())
        assert np.abs(mine[2].cpu().numpy() - theirs[2].cpu().numpy()).max() <= 1e-6
    # fused expansion and masked policy through the small-batch form
    n = 50
    sl = slice(0, n)
    legal = torch.from_numpy(pos256["legal"][sl].view(np.int64).copy()).cuda()
    got = {}
    for form in (1, 0):
        enc.set_one_board(form)
        pri, mov, ne, val = (t.clone() for t in enc.forward_priors(*inputs(pos256, sl), legal, 96, logits=True))
        got[form] = (pri, mov, ne, val, enc.policy_out.clone())
    for a, b in zip(got[1], got[0]):
        assert torch.equal(a.view(torch.uint8) if a.dtype is torch.half else a, b.view(torch.uint8) if b.dtype is torch.half else b)
    enc.set_one_board(1)
    enc.close()


def test_fp16_arithmetic_is_bit_identical_to_the_reference_kernel(pos256, pos4096):
    """`FusedEncoder(net, int8=False)`: the reference's default arithmetic, every weight GEMM fp16
    x fp16.  tcgen05 `kind::f16` with fp16 accumulators carries the bits of the reference's
    fp16-accumulate mma.sync, and the ff2 accumulators run through the four hidden chunks as the
    reference's do, so every stage and every output is equal to the bit."""
    if not R.available("A_f16"):
        pytest.skip("slabs missing")
    enc, ref = product(SETS["A"], int8=False), R.RefKernel("A_f16")
    assert ref.quant == 0 and enc.quant == 0 and enc.label.startswith("fp16")
    sl = slice(0, 200)
    for stage in (9, 1, 5, 6, 7, 4, 2, 3, 8):
        got = enc.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        want = ref.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        assert same_bits(got, want), stage
    for pos, sl in ((pos256, slice(3, 3 + 77)), (pos4096, slice(0, 4096))):
        (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos, sl)
        assert same_bits(pol, rpol) and same_bits(pro, rpro) and np.abs(val - rval).max() <= 1e-6
    enc.close()


@pytest.mark.parametrize("scheme,name,quant,fmt", [("ffn", "B_int8_ffn", 2, "int8_ffn"),
                                                   ("ffn+qkv", "B_int8_ffn_qkv", 4, "int8_ffn_qkv")])
def test_partial_int8_schemes_are_bit_identical(scheme, name, quant, fmt, pos256, pos4096):
    """`int8_scheme="ffn"` (the reference's quant 2): the FFN in s8/u8 as in the shipped scheme,
    QKV and out-projection in fp16 as in the default arithmetic; `"ffn+qkv"` (quant 4): QKV in
    s8 as well, only the out-projection in fp16.  Each GEMM carries the reference's bits on its
    own, so do the mixtures."""
    if not R.available(name):
        pytest.skip("slabs missing")
    enc, ref = product(SETS["B"], int8=True, int8_scheme=scheme), R.RefKernel(name)
    assert ref.quant == quant and enc.quant == quant and enc.label.startswith("int8 FFN")
    sl = slice(0, 200)
    for stage in (9, 1, 5, 6, 7, 4, 2, 3, 8):
        got = enc.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        want = ref.forward_stage(*inputs(pos256, sl), stage).cpu().numpy()
        assert same_bits(got, want), stage
    for pos, sl in ((pos256, slice(5, 5 + 91)), (pos4096, slice(0, 4096))):
        (pol, pro, val), (rpol, rpro, rval) = run_both(enc, ref, pos, sl)
        assert same_bits(pol, rpol) and same_bits(pro, rpro) and np.abs(val - rval).max() <= 1e-6
    # and against the CPU restatement of the same mixture, at the quantised-path tolerance
    from brokefish_b200.nn.model import seeded_state
    w = O.prepare({k: v.numpy() for k, v in seeded_state(**SETS["B"]).items()}, fmt=fmt)
    n = 48
    opol, opro, oval = O.forward(w, pos256["boards"][:n], pos256["control"][:n], pos256["rep"][:n])[:3]
    enc.exact_rsqrt = True
    pol, pro, val = [t.cpu().numpy().copy() for t in enc.forward_full(*inputs(pos256, slice(0, n)))]
    d = np.abs(pol.astype(np.float32) - opol.astype(np.float32)).max()
    print(f"{scheme} arm vs CPU restatement: max|dlogit| {d:.4f} of {np.abs(opol.astype(np.float32)).max():.3f}")
    assert d <= rel_tol(opol, 2e-2)
    enc.close()


def test_timing_report(pos4096):
    """Not a bar: prints both kernels' device time on the 4096-position batch (CUDA events, 5
    warm-ups, 20 timed launches each) so the summary under profiles/ can be reproduced with
    ``pytest tests/test_gpu_reference_kernel.py -m gpu -s -k timing``."""
    if not R.available("A_int8"):
        pytest.skip("slabs missing")
    args = inputs(pos4096, slice(0, 4096))

    def ms(fn, n=20):
        for _ in range(5):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(n):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / n

    enc = product(SETS["A"])
    rows = [("product int8", ms(lambda: enc.forward_full(*args)))]
    enc.close()
    enc = product(SETS["A"], fp8=True)
    rows.append(("product e4m3 FFN", ms(lambda: enc.forward_full(*args))))
    enc.close()
    enc = product(SETS["A"], int8=False)
    rows.append(("product fp16", ms(lambda: enc.forward_full(*args))))
    enc.close()
    for tag, label in (("A_int8", "reference kernel int8 (all four GEMMs, two boards per CTA)"),
                       ("A_f16", "reference kernel fp16"), ("A_e4m3", "reference kernel e4m3 FFN")):
        if R.available(tag):
            ref = R.RefKernel(tag)
            rows.append((label, ms(lambda: ref.forward_full(*args))))
    for label, t in rows:
        print(f"{label:64s} {t:7.3f} ms / 4096 positions  {4096 / t * 1e3:12.0f} pos/s")
    assert all(t > 0 for _, t in rows)
