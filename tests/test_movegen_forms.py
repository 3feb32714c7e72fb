"""The thread-per-board move generator's two forms, compiled for the host: `board_moves`, which goes by the
slots pieces start in, gives the words of `board_moves_any`, which takes any board, on every kind of board it
can be handed -- played, promoted, rearranged, malformed."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import GOLDEN, ROOT

STUBS = r"""
#include <stdint.h>
#include <algorithm>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __noinline__
using std::min;
struct ulonglong2 { unsigned long long x, y; };
inline int __popcll(unsigned long long v) { return __builtin_popcountll(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
inline unsigned __byte_perm(unsigned x, unsigned y, unsigned s) {
    const unsigned long long v = ((unsigned long long)y << 32) | x;
    unsigned r = 0;
    for (int i = 0; i < 4; ++i) r |= (unsigned)((v >> (8 * ((s >> (4 * i)) & 7))) & 255) << (8 * i);
    return r;
}
inline unsigned long long __brevll(unsigned long long v) {
    unsigned long long r = 0;
    for (int i = 0; i < 64; ++i) if ((v >> i) & 1) r |= 1ull << (63 - i);
    return r;
}
"""

MAIN = r"""
// boards whose words or check flags differ; `fast` gets the words, `by_slot` which form made them
extern "C" long compare(const unsigned short* boards, const short* control, long n, unsigned long long* fast, unsigned char* by_slot) {
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        unsigned my[17];
        unsigned long long own[16], any[32], *all = fast + 32 * i;
        std::memcpy(my, boards + 32 * i, 64);
        const bool black = control[i] < 0;
        bool slots;
        const bool a = board_moves(my, black, own, all, kMoveTables, slots), b = board_moves_any(my, black, any);
        if (slots) {
            std::memset(all, 0, 256);
            std::memcpy(all + (black ? 16 : 0), own, 128);
        }
        by_slot[i] = slots;
        bad += a != b || std::memcmp(all, any, 256) != 0;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def compare(tmp_path_factory):
    text = open(os.path.join(ROOT, "brokefish_b200", "csrc", "bf_movegen.cuh")).read()
    cut = lambda a, b: text[text.index(a):text.index(b)]
    parts = [cut("constexpr unsigned long long kFileA", "__device__ __forceinline__ unsigned long long warp_or"),
             cut("__device__ __forceinline__ unsigned long long knight_pattern", "// Squares seen from `sq` along the rook"),
             cut("template <int kShift>", "// Castling rights KQkq as four bits of a board held by one thread")]
    source = re.sub(r'unsigned lo, hi;\s*asm\("shl.*?\n\s*asm\(.*?\n',
                    "unsigned lo = s < 32u ? 1u << s : 0u, hi = s - 32u < 32u ? 1u << (s - 32u) : 0u;\n", "".join(parts), flags=re.S)
    source = re.sub(r"asm volatile\([^;]*;", "", source)
    folder = tmp_path_factory.mktemp("forms")
    (folder / "forms.cpp").write_text(STUBS + source + MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w", str(folder / "forms.cpp"), "-o", str(folder / "forms.so")],
                   check=True)
    lib = ctypes.CDLL(str(folder / "forms.so"))
    lib.compare.restype = ctypes.c_long

    def run(boards, control):
        b, c = np.ascontiguousarray(boards, dtype=np.uint16), np.ascontiguousarray(control, dtype=np.int16)
        words, slots = np.zeros((len(c), 32), np.uint64), np.zeros(len(c), np.uint8)
        at = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        return lib.compare(at(b), at(c), ctypes.c_long(len(c)), at(words), at(slots)), words, slots
    return run


def test_played_boards(compare, pos4096):
    gold = np.load(os.path.join(GOLDEN, "ref_movegen.npz"))
    bad, words, slots = compare(pos4096["boards"], pos4096["control"])
    assert bad == 0 and np.array_equal(words, pos4096["legal"].view(np.uint64)) and slots.all()
    bad, words, slots = compare(gold["fen_boards"], gold["fen_control"])
    assert bad == 0 and np.array_equal(words, gold["fen_legal"])


SLOT, PAWN_SLOT = np.arange(32), np.arange(32) % 16 < 8


def distinct_squares(rng, b):
    return (b & ~np.uint16(63)) | np.argsort(rng.random((len(b), 64)), 1)[:, :32].astype(np.uint16)


def promoted(rng, b, c):
    where = PAWN_SLOT & (rng.random(b.shape) < 0.3) & ((b >> 11) & 1 == 0)
    return np.where(where, (b & ~np.uint16(0x3C0)) | (rng.integers(1, 5, b.shape) << 6) | (rng.integers(0, 2, b.shape) << 9), b)


def scattered(rng, b, c):
    b = np.where(rng.random(b.shape) < 0.5, 0x800, distinct_squares(rng, b)) ^ ((rng.random(b.shape) < 0.2) * 0x200)
    where = PAWN_SLOT & (rng.random(b.shape) < 0.1) & ((b >> 11) & 1 == 0)
    return np.where(where, (b & ~np.uint16(0x1C0)) | (rng.integers(0, 8, b.shape) << 6), b)


def pawns_side_by_side(rng, b, c):
    """Flagged pawns beside the mover's on the rank where en passant is taken."""
    b = b.copy()
    for i in range(len(b)):
        own, rank, files = (0, 4, rng.permutation(8)) if c[i] > 0 else (16, 3, rng.permutation(8))
        for j in range(4):
            b[i, own + j] = rank * 8 + files[2 * j] | (0x400 if own else 0)
            b[i, 16 - own + j] = rank * 8 + files[2 * j + 1] | (0 if own else 0x400) | (0x200 if rng.random() < 0.4 else 0)
    return b


KINDS = {
    "promoted": (promoted, True),
    "distinct squares": (lambda rng, b, c: np.where(rng.random(b.shape) < 0.4, 0x800, distinct_squares(rng, b)), True),
    "scattered, flagged, of any type": (scattered, None),
    "en passant": (pawns_side_by_side, None),
    "some words changed": (lambda rng, b, c: np.where(rng.random(b.shape) < 0.03, b ^ rng.integers(0, 4096, b.shape), b), None),
    "upper bits, captured with a type": (lambda rng, b, c: np.where(rng.random(b.shape) < 0.1, b | 0x800, b) |
                                         (rng.integers(0, 16, b.shape) << 12), True),
    "slots shuffled": (lambda rng, b, c: rng.permuted(b, axis=1), False),
    "any words": (lambda rng, b, c: rng.integers(0, 65536, b.shape), False),
}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("turned", [1, -1])
def test_boards_of_every_kind(kind, turned, compare, pos4096):
    make, by_slot = KINDS[kind]
    rng = np.random.default_rng(len(kind))
    control = pos4096["control"] * turned
    boards = make(rng, pos4096["boards"].astype(np.uint16), control)
    bad, _, slots = compare(boards, control)
    assert bad == 0
    # the boards take the form that is meant for them
    if by_slot is not None:
        assert (slots != 0).mean() > 0.99 if by_slot else (slots != 0).mean() < 0.01
    else:
        assert slots.any() and not slots.all()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [12288, 12289, 31744, 31745, 45056, 45057, 163841, 327681])
def test_either_side_of_the_lines_between_a_launch_s_forms(n, pos4096):
    from test_movegen import test_both_forms_of_the_engine_kernels_agree_at_every_size as agree
    agree(n, pos4096)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [34816, 34817, 40001])
def test_a_random_ply_either_side_of_its_line(n, pos4096):
    """The same boards with the same draws in batches of 4096 (eight lanes per board) and in one."""
    import torch
    from brokefish_b200 import _native
    L, at = _native.lib(), lambda t: ctypes.c_void_p(t.data_ptr())
    place = torch.arange(n) % 4096
    start = [torch.from_numpy(np.ascontiguousarray(pos4096[k])).view(torch.int16)[place].cuda() for k in ("boards", "control")]
    start.append(torch.from_numpy(pos4096["legal"].view(np.int64))[place].cuda())
    gen = torch.Generator().manual_seed(n)
    draw, promo = torch.rand(n, generator=gen).cuda(), torch.randint(0, 4, (n,), generator=gen).to(torch.int8).cuda()

    def ply(step):
        b, c, m = (t.clone() for t in start)
        move = torch.empty(n, dtype=torch.int32, device="cuda")
        for lo in range(0, n, step):
            part = [t[lo:lo + step] for t in (b, c, m, draw, promo)]
            _native.check(L.bf_random_ply(0, *(at(t) for t in part), len(part[0]), at(move[lo:]),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "bf_random_ply")
        return b, c, m, move
    for got, want in zip(ply(n), ply(4096)):
        assert torch.equal(got, want)
