"""The barrier schedule of the one- and two-board tiles, on the CPU: the kernel's own row-warp and MMA-issue
functions are compiled for the host with their arithmetic taken out, and what is left -- waits, arrivals,
commits -- is recorded.  A parity wait tells a phase only from the one before it, so on every barrier the
waiting side has to wait for each phase, in order, and the other side has to complete just those."""
import os
import re
import subprocess

import pytest

from conftest import ROOT

ARITHMETICS = ["kArInt8", "kArE4M3", "kArF16", "kArI8Ffn", "kArI8Qkv"]
LAYERS, TILES = 3, 3

STUBS = r"""
#include <cstdint>
#include <cstdio>
#define __device__
#define __host__
#define __forceinline__ inline
struct uint4 { uint32_t x, y, z, w; };
struct Scale { float scale = 1, inverse = 1; };
struct Bias { uint4 lo, hi; };
struct Issue { uint32_t smem, tmem; volatile int* abort_flag; uint32_t i, a, h; };
struct Row { int lane, q, s; uint32_t smem, tm; volatile int* abort_flag; uint64_t one2; uint32_t layers, tiles, h;
             uint32_t a() const { return 0; } };
enum { kKindI8, kKindF16, kKindF8, kAccPlain, kAccInt, kAccFloat, kAccS32, kAccF16, kAccF32, kFmtS8, kFmtU8, kFmtF16, kFmtE4M3,
       kErrRowAcc, kErrMmaWeights, kErrMmaOperand, LP_B_QKV = 0, LP_SW_QKV, LP_B_O, LP_SW_O, LP_B_FF1, LP_SW_FF1, LP_B_FF2,
       LP_SW_FF2, SM_MAX, SM_A, kHeadA, kHeadStages = 4, kStage = 0 };
enum { kArInt8, kArE4M3, kArF16, kArI8Ffn, kArI8Qkv };
template <int> struct Cfg { static constexpr bool kQkvF16 = false, kOutF16 = false; static constexpr int kQkvSlabs = 2, kOutSlabs = 2, kFfnSlabs = 2; };
template <int> struct Map { static constexpr uint32_t kStages = 4, SM_RING = 0, SM_H = 0; };
struct Any { template <class T> operator T() const { return T(); } };
uint32_t bar(uint32_t, int i) { return i; }
void say(const char* what, int b, int parity) { if (b >= B_ACC) std::printf("%s %d %d\n", what, b, parity); }
// (barriers that both SMs of a pair arrive at are waited for across them, no others)
void check(bool across, int b) { if (across != (b < B_EMPTY || (b >= B_A && b < B_MAX))) std::printf("scope %d 0\n", b); }
bool mbar_wait(uint32_t b, uint32_t parity, volatile int*, int) { check(false, b); say("wait", b, parity); return true; }
bool mbar_wait_cluster(uint32_t b, uint32_t parity, volatile int*, int) { check(true, b); say("wait", b, parity); return true; }
void mbar_arrive_first(uint32_t b) { say("done", b, 0); }
void tc_commit_pair(uint32_t b) { say("done", b, 0); }
bool elect_one() { return true; }
template <class... T> constexpr uint32_t umma_idesc(T...) { return 0; }
template <int NB, class F> void each_piece(uint32_t, F&&) {}
#define NOTHING(name) template <class... T> Any name(T&&...) { return Any(); }
#define NOTHING_NB(name) template <int NB, class... T> Any name(T&&...) { return Any(); }
NOTHING(__syncwarp) NOTHING(tc_fence_after) NOTHING(tc_fence_before) NOTHING(fence_proxy_async_smem)
NOTHING(umma_pair_f16) NOTHING(umma_pair_f8) NOTHING(umma_pair_i8) NOTHING(named_bar_sync) NOTHING(pair_sync) NOTHING(lds_f) NOTHING(load_bias)
NOTHING(sts128) NOTHING(load_query) NOTHING(scores) NOTHING(softmax) NOTHING(weighted_values) NOTHING(store_outputs)
NOTHING(max_to) NOTHING(scale_s8) NOTHING(scale_u8) NOTHING(scale_e4m3) NOTHING_NB(amax_h2) NOTHING_NB(board_sync)
NOTHING_NB(store_operand16)
template <int NB, bool kE4M3 = false, class... T> void store_operand8(T&&...) {}
template <bool kRelu, int kAcc, class... T> void descale16(T&&...) {}
uint32_t head_off(int, int) { return 0; }
uint64_t umma_desc_k128(uint32_t) { return 0; }
uint4 make_uint4(uint32_t, uint32_t, uint32_t, uint32_t) { return {}; }
uint4 lds128(uint32_t) { return {}; }
struct Half2 {};
Half2 as_h2(uint32_t) { return {}; }
Half2 __hadd2(Half2, Half2) { return {}; }
uint32_t as_u32(Half2) { return 0; }
uint64_t pk2(float, float) { return 0; }
uint64_t mul2(uint64_t, uint64_t) { return 0; }
uint64_t fma2(uint64_t, uint64_t, uint64_t) { return 0; }
uint64_t h2_to_f2(uint32_t) { return 0; }
uint32_t f2_to_h2(uint64_t) { return 0; }
float __uint_as_float(uint32_t) { return 0; }
"""

MAIN = r"""
template <int NB> void rows() {
    Row c = {};
    uint32_t x[8 * NB] = {};
    for (int tile = 0; tile < TILES; ++tile, ++c.tiles) {
        for (int layer = 0; layer < LAYERS; ++layer, ++c.layers) {
            publish(c, B_A);
            attention_block<NB, AR>(c, 0, 1.f, 0u, x);
            publish(c, B_A);
            if constexpr (AR == kArF16) ffn_block_f16<NB>(c, 0, x);
            else ffn_block<NB, AR>(c, 0, 1.f, x);
        }
        publish(c, B_A);
        wait_acc<AR>(c, 0, 0);
    }
}
int main() {
    std::puts("rows"); rows<BOARDS>();
    std::puts("issue");
    Issue st = {};
    for (int tile = 0; tile < TILES; ++tile) issue_tile<BOARDS, AR>(st, LAYERS);
}
"""


def definition(text, start):
    """The definition that begins with `start`, its template line included."""
    at = text.index(start)
    before = text.rfind("\n", 0, at - 1) + 1
    if text[before:at].startswith("template"):
        at = before
    depth, i = 0, text.index("{", at)
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[at:i] + (";" if start.startswith("struct") else "")


@pytest.fixture(scope="module")
def source():
    text = open(os.path.join(ROOT, "brokefish_b200", "csrc", "bf_encoder_ws.cuh")).read()
    inline = "__device__ __forceinline__ void "
    parts = [re.search(r"enum \{ B_FULL.*?\};", text).group(0), STUBS, definition(text, "struct Own"),
             definition(text, "__host__ __device__ constexpr uint32_t completions")]
    parts += [definition(text, inline + name + "(") for name in
              ("wait_acc", "publish", "stage_qkv", "attention_block", "ffn_block", "ffn_block_f16", "issue_unit", "issue_wait",
               "issue_tile")]
    return "\n".join(parts + [MAIN])


@pytest.mark.parametrize("boards", [1, 2])
@pytest.mark.parametrize("arithmetic", ARITHMETICS)
def test_every_phase_is_waited_for(arithmetic, boards, source, tmp_path):
    src, exe = tmp_path / "schedule.cpp", tmp_path / "schedule"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-w", f"-DAR={arithmetic}", f"-DBOARDS={boards}", f"-DLAYERS={LAYERS}",
                    f"-DTILES={TILES}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows, issue = (part.split("\n") for part in out.replace("rows\n", "").split("issue\n"))
    waits, done = {}, {}
    for lines in (rows, issue):
        for line in filter(None, lines):
            what, b, parity = line.split()
            assert what != "scope", f"barrier {b} is waited for at the wrong scope"
            if what == "wait":
                waits.setdefault(int(b), []).append(int(parity))
            else:
                done[int(b)] = done.get(int(b), 0) + 1
    assert set(waits) == set(done) and len(done) >= 7          # four slots, the operand, two hidden pairs
    for b, parities in waits.items():
        assert parities == [i & 1 for i in range(done[b])], b


def test_what_crosses_between_sms_is_ordered_at_cluster_scope():
    """At the default scope, the CTA's, an arrival and a wait order nothing between two SMs."""
    text = open(os.path.join(ROOT, "brokefish_b200", "csrc", "bf_ptx.cuh")).read()
    arrive = definition(text, "__device__ __forceinline__ void mbar_arrive_cluster(")
    assert arrive.index("fence.release.sync_restrict::shared::cta.cluster") < arrive.index("mbarrier.arrive.relaxed.cluster.shared::cluster")
    wait = definition(text, "__device__ __forceinline__ bool mbar_wait_cluster(")
    assert wait.index("mbar_wait<0, true>") < wait.index("fence.acquire.sync_restrict::shared::cluster.cluster")
    assert "mbarrier.try_wait.parity.relaxed.cluster" in definition(text, "__device__ __forceinline__ uint32_t mbar_try_wait(")


# ---- the weight ring ----

RING = r"""
#include <vector>
struct Params { const uint8_t *wstream = nullptr, *lparams = nullptr; int n_layers = LAYERS, after_waves = 0; };
enum { kErrProducer = 100, kQStage = 0, kRStage = 0, kHeadStage = 16384, kLparamStride = 0, SM_PAR = 0 };
template <int AR_> struct RingCfg : Cfg<AR_> { static constexpr int kLayerStream = 0; };
#define Cfg RingCfg
static std::vector<int> sent(64), waited(64);
static bool wrong = false;
bool ring_wait(uint32_t b, uint32_t parity, volatile int*, int) {
    if (b >= B_EMPTY && b < B_ACC) wrong |= ((unsigned)(waited[b - B_EMPTY]++) & 1u) != parity;
    return true;
}
void ring_send(uint32_t b, uint32_t) { if (b < B_EMPTY) ++sent[b - B_FULL]; }
template <class... T> void bulk_g2s(T&&...) {}
void previous_grid_wait() {}
void next_grid_may_start() {}
long long clock64() { return 1ll << 40; }
#define mbar_wait ring_wait
#define mbar_arrive_expect_tx ring_send
"""

RING_MAIN = r"""
int main() {
    volatile int abort_flag = 0;
    Params p;
    producer<AR>(0, &abort_flag, p, TILES, RANK);
    for (int k = 0; k < B_EMPTY; ++k)
        if (sent[k] != waited[k]) { std::printf("place %d: sent %d times, waited for %d\n", k, sent[k], waited[k]); return 1; }
    if (wrong) std::puts("a wait's parity is not the next phase's");
    return wrong;
}
"""


@pytest.mark.parametrize("tiles", [0, 1, 3])
@pytest.mark.parametrize("stages", [6, 8])
@pytest.mark.parametrize("arithmetic", ["kArInt8", "kArF16"])
def test_the_weight_ring_is_drained(arithmetic, stages, tiles, tmp_path):
    """Each stage's consumption arrives at a barrier of both SMs of a pair.  The producer waits for every one of
    them, the last ones too: none may be on its way when the shared memory is another grid's."""
    text = open(os.path.join(ROOT, "brokefish_b200", "csrc", "bf_encoder_ws.cuh")).read()
    stubs = STUBS.replace("kStages = 4", f"kStages = {stages}")
    parts = [definition(text, start) for start in ("__device__ __forceinline__ void drain(", "__device__ __forceinline__ void producer(")]
    main = "\n".join([re.search(r"enum \{ B_FULL.*?\};", text).group(0), stubs, RING, *parts, RING_MAIN])
    for rank in (0, 1):
        src, exe = tmp_path / "ring.cpp", tmp_path / f"ring{rank}"
        src.write_text(main)
        subprocess.run(["g++", "-std=c++17", "-w", f"-DAR={arithmetic}", f"-DLAYERS={LAYERS}", f"-DTILES={tiles}", f"-DRANK={rank}",
                        str(src), "-o", str(exe)], check=True)
        out = subprocess.run([str(exe)], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout
