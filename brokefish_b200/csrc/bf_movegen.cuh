// Legal-move generation and move application for the 32-slot piece-list board, in two forms:
// `legal_word`, one warp per board with lane = slot (what the evaluator's expansion warp calls),
// and the stand-alone kernels further down, eight lanes per board (launches that do not fill the
// GPU) or one thread per board (the large ones).
//
// The contract of the reference's engine (brokefish/env/torch_impl.py:254-291, csrc/movegen.cuh):
// `mask [n,32]` 64-bit words, bit s of word p set when the piece in slot p may legally move to
// square s, and `in_check [n]` for the side to move.  A promotion is one bit (the type travels
// beside the move); castling is the king's two-square move; en passant is a pawn's diagonal move
// onto an empty square.
//
// Piece word (brokefish/env/torch_impl.py:40-47): bits 0-5 square (rank * 8 + file), 6-8 type
// (0 pawn, 1 knight, 2 bishop, 3 rook, 4 queen, 5 king), bit 9 "special" (king, rook: has moved;
// pawn: has just made its double step), bit 10 colour (1 black), bit 11 captured.  The control
// word's sign is the side to move (negative: black).
//
// Method of the warp form: bitboards built with warp-wide OR reductions; every enemy lane contributes the squares
// its piece attacks with the mover's king lifted off the board (king moves and castling avoid
// their union); the enemy lanes that attack the king are the checkers (one checker: the other
// pieces may only capture it or step between; two: only the king moves); every lane walks the
// line from the king to its own piece, which finds the pieces that shield the king from a slider
// (they move only along that line) and, for a checking slider, the squares between.  Only en
// passant, which takes two pieces off one rank at once, is tested on the position after the
// move.  This decides what the reference decides by replaying each move and building the
// opponent's control map (torch_impl.py:266-290).
#pragma once
#include <stdint.h>

namespace bfmg {

// These kernels are launched before the grid before them in the stream has quite ended: they wait for it before they
// touch its memory.  (No __restrict__ on what they read: the compiler may move a load from memory that it takes to
// be constant above the wait.)  Legal words by a thread per board let the grid after them start when a block
// has made its words; the others say nothing, and the next grid starts as theirs drains: its blocks, placed among the
// ones that still run, leave the SMs uneven (a move with words and key of 4096 boards 9.6 us a launch instead of 6.6).
__device__ __forceinline__ void after_previous_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_grid_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

constexpr unsigned long long kFileA = 0x0101010101010101ull, kFileH = kFileA << 7;
constexpr unsigned kFull = 0xffffffffu;
enum { PAWN = 0, KNIGHT = 1, BISHOP = 2, ROOK = 3, QUEEN = 4, KING = 5 };

__device__ __forceinline__ unsigned long long warp_or(unsigned long long v) {
    const unsigned lo = __reduce_or_sync(kFull, static_cast<unsigned>(v));
    const unsigned hi = __reduce_or_sync(kFull, static_cast<unsigned>(v >> 32));
    return (static_cast<unsigned long long>(hi) << 32) | lo;
}
__device__ __forceinline__ unsigned long long knight_pattern(unsigned long long b) {
    const unsigned long long l1 = (b >> 1) & ~kFileH, l2 = (b >> 2) & ~(kFileH | (kFileH >> 1));
    const unsigned long long r1 = (b << 1) & ~kFileA, r2 = (b << 2) & ~(kFileA | (kFileA << 1));
    const unsigned long long h1 = l1 | r1, h2 = l2 | r2;
    return (h1 << 16) | (h1 >> 16) | (h2 << 8) | (h2 >> 8);
}
__device__ __forceinline__ unsigned long long king_pattern(unsigned long long b) {
    const unsigned long long row = b | ((b >> 1) & ~kFileH) | ((b << 1) & ~kFileA);
    return (row | (row << 8) | (row >> 8)) & ~b;
}
// One sliding piece along one line without loops or fills: on the line's squares other than the
// piece's own, subtracting the piece's bit from the occupancy flips exactly the squares up to and
// including the first occupied one above it; the same on the bit-reversed board gives the squares
// below it (the method published as o^(o-2r) and, with a reversed board, as hyperbola quintessence).
__device__ __forceinline__ unsigned long long line_attacks(unsigned long long s, unsigned long long occ,
                                                           unsigned long long line_ex) {
    const unsigned long long o = occ & line_ex;
    const unsigned long long up = o - s;
    const unsigned long long down = __brevll(__brevll(o) - __brevll(s));
    return (up ^ down) & line_ex;
}
// The rank, file and two diagonals through a square, without the square itself.
__device__ __forceinline__ unsigned long long rank_ex(int sq) { return (0xFFull << (sq & 56)) ^ (1ull << sq); }
__device__ __forceinline__ unsigned long long file_ex(int sq) { return (kFileA << (sq & 7)) ^ (1ull << sq); }
__device__ __forceinline__ unsigned long long diag_ex(int sq) {
    const int d = (sq >> 3) - (sq & 7);
    return (d >= 0 ? 0x8040201008040201ull << (8 * d) : 0x8040201008040201ull >> (-8 * d)) ^ (1ull << sq);
}
__device__ __forceinline__ unsigned long long anti_ex(int sq) {
    const int d = (sq >> 3) + (sq & 7) - 7;
    return (d >= 0 ? 0x0102040810204080ull << (8 * d) : 0x0102040810204080ull >> (-8 * d)) ^ (1ull << sq);
}
// Squares seen from `sq` along the rook (diag = false) or bishop (diag = true) lines, each ray
// ending on and including its first occupied square.
__device__ __forceinline__ unsigned long long rays(int sq, unsigned long long occ, bool diag) {
    const unsigned long long b = 1ull << sq;
    return diag ? line_attacks(b, occ, diag_ex(sq)) | line_attacks(b, occ, anti_ex(sq))
                : line_attacks(b, occ, rank_ex(sq)) | line_attacks(b, occ, file_ex(sq));
}

// The opponent's pieces by the way they attack.
struct Enemy {
    unsigned long long pawns, knights, diag, line, king;
    bool black;                 // the opponent's colour
};

__device__ __forceinline__ bool attacked(int sq, unsigned long long occ, const Enemy& e) {
    const unsigned long long b = 1ull << sq;
    if (knight_pattern(b) & e.knights) return true;
    if (king_pattern(b) & e.king) return true;
    // a black pawn stands one rank above the square it attacks, a white pawn one rank below
    const unsigned long long from = e.black ? (((b << 7) & ~kFileH) | ((b << 9) & ~kFileA))
                                            : (((b >> 7) & ~kFileA) | ((b >> 9) & ~kFileH));
    if (from & e.pawns) return true;
    if (rays(sq, occ, false) & e.line) return true;
    return (rays(sq, occ, true) & e.diag) != 0ull;
}
__device__ __forceinline__ Enemy without(const Enemy& e, unsigned long long gone) {
    Enemy r = e;
    r.pawns &= ~gone; r.knights &= ~gone; r.diag &= ~gone; r.line &= ~gone; r.king &= ~gone;
    return r;
}

// Warp-collective: every lane passes its slot's piece word; returns this slot's legal-target
// word.  `in_check` (same value on every lane) says whether the side to move is in check.
__device__ __forceinline__ unsigned long long legal_word(unsigned word, int control, bool& in_check) {
    const bool black = control < 0;
    const bool live = ((word >> 11) & 1u) == 0u;
    const bool is_black = (word >> 10) & 1u;
    const bool special = (word >> 9) & 1u;
    const int type = (word >> 6) & 7;
    const int sq = word & 63;
    const bool mine = live && (is_black == black);
    const bool theirs = live && (is_black != black);
    const unsigned long long bb = live ? (1ull << sq) : 0ull;

    const unsigned long long occ = warp_or(bb);
    const unsigned long long own = warp_or(mine ? bb : 0ull);
    const unsigned long long opp = occ & ~own;
    Enemy e;
    e.black = !black;
    e.pawns = warp_or(theirs && type == PAWN ? bb : 0ull);
    e.knights = warp_or(theirs && type == KNIGHT ? bb : 0ull);
    e.diag = warp_or(theirs && (type == BISHOP || type == QUEEN) ? bb : 0ull);
    e.line = warp_or(theirs && (type == ROOK || type == QUEEN) ? bb : 0ull);
    e.king = warp_or(theirs && type == KING ? bb : 0ull);
    const unsigned long long ep_pawns = warp_or(theirs && type == PAWN && special ? bb : 0ull);
    const unsigned long long fresh_rooks = warp_or(mine && type == ROOK && !special ? bb : 0ull);
    const unsigned long long my_king = warp_or(mine && type == KING ? bb : 0ull);
    const int king_sq = my_king ? __ffsll(static_cast<long long>(my_king)) - 1 : 0;
    const int rank = sq >> 3, file = sq & 7;

    // ---- what the opponent attacks, with the mover's king lifted off the board (so that a
    //      square behind the king on a checking line counts as attacked) ----
    unsigned long long att = 0ull;
    if (theirs) {
        const unsigned long long occ_nk = occ & ~my_king;
        if (type == PAWN)
            att = is_black ? (((bb >> 9) & ~kFileH) | ((bb >> 7) & ~kFileA))
                           : (((bb << 7) & ~kFileH) | ((bb << 9) & ~kFileA));
        else if (type == KNIGHT) att = knight_pattern(bb);
        else if (type == KING) att = king_pattern(bb);
        else {
            if (type == BISHOP || type == QUEEN) att |= rays(sq, occ_nk, true);
            if (type == ROOK || type == QUEEN) att |= rays(sq, occ_nk, false);
        }
    }
    const unsigned long long danger = warp_or(att);
    in_check = (danger & my_king) != 0ull;
    const unsigned checkers = __ballot_sync(kFull, theirs && (att & my_king) != 0ull);

    // ---- the line from the king to this piece, when the piece is the first one met on a rank,
    //      file or diagonal through the king: `line_to_me` = squares after the king up to and
    //      including the piece, `beyond` = the next piece on the same ray, `line` = everything
    //      walked, from the king's neighbour to that next piece ----
    unsigned long long line = 0ull, line_to_me = 0ull, beyond = 0ull;
    bool first_on_ray = false, ray_diag = false;
    if (live && my_king != 0ull && bb != my_king) {
        const int kr = king_sq >> 3, kf = king_sq & 7;
        const int dr = rank - kr, df = file - kf;
        const bool aligned = (dr == 0) != (df == 0) || (dr != 0 && (dr == df || dr == -df));
        if (aligned) {
            const int sr = (dr > 0) - (dr < 0), sf = (df > 0) - (df < 0);
            ray_diag = sr != 0 && sf != 0;
            int r = kr + sr, f = kf + sf;
            bool past = false;
            while (r >= 0 && r < 8 && f >= 0 && f < 8) {
                const unsigned long long bit = 1ull << (r * 8 + f);
                line |= bit;
                if (!past) line_to_me |= bit;
                if (occ & bit) {
                    if (!past) {
                        if (bit != bb) break;          // something stands between the king and this piece
                        past = first_on_ray = true;
                    } else {
                        beyond = bit;
                        break;
                    }
                }
                r += sr; f += sf;
            }
        }
    }
    // one checker: the other pieces may only capture it or step between it and the king
    unsigned long long target_mask = ~0ull;
    const int n_checkers = __popc(checkers);
    {
        const bool slider = type == BISHOP || type == ROOK || type == QUEEN;
        const unsigned long long blk = (slider && first_on_ray) ? line_to_me : bb;
        const int c = checkers ? __ffs(checkers) - 1 : 0;
        const unsigned lo = __shfl_sync(kFull, static_cast<unsigned>(blk), c);
        const unsigned hi = __shfl_sync(kFull, static_cast<unsigned>(blk >> 32), c);
        if (n_checkers == 1) target_mask = (static_cast<unsigned long long>(hi) << 32) | lo;
        else if (n_checkers > 1) target_mask = 0ull;
    }
    if (!mine) return 0ull;

    // ---- pseudo-legal targets ----
    unsigned long long cand = 0ull, ep_target = 0ull;
    if (type == KNIGHT) {
        cand = knight_pattern(bb);
    } else if (type == KING) {
        cand = king_pattern(bb) & ~danger;
        // castling: neither the king's square nor the one it crosses nor the one it lands on may
        // be attacked (on the first rank nothing the rook's jump uncovers or covers changes that)
        if (!special && !in_check) {
            const int row = black ? 56 : 0;
            if ((fresh_rooks >> (row + 7)) & 1ull)
                if (((occ >> (row + 5)) & 3ull) == 0ull && ((danger >> (row + 5)) & 3ull) == 0ull)
                    cand |= 1ull << (row + 6);
            if ((fresh_rooks >> row) & 1ull)
                if (((occ >> (row + 1)) & 7ull) == 0ull && ((danger >> (row + 2)) & 3ull) == 0ull)
                    cand |= 1ull << (row + 2);
        }
        return cand & ~own;
    } else if (type == PAWN) {
        const int up = black ? -8 : 8;
        const int f1 = sq + up;
        if (f1 >= 0 && f1 < 64 && !((occ >> f1) & 1ull)) {
            cand |= 1ull << f1;
            const bool start = black ? rank == 6 : rank == 1;
            if (start && !((occ >> (f1 + up)) & 1ull)) cand |= 1ull << (f1 + up);
        }
        if (f1 >= 0 && f1 < 64) {
            if (file > 0) cand |= (1ull << (f1 - 1)) & opp;
            if (file < 7) cand |= (1ull << (f1 + 1)) & opp;
            // en passant: an enemy pawn that has just made its double step stands beside us
            if (rank == (black ? 3 : 4)) {
                if (file > 0 && ((ep_pawns >> (sq - 1)) & 1ull)) ep_target |= 1ull << (f1 - 1);
                if (file < 7 && ((ep_pawns >> (sq + 1)) & 1ull)) ep_target |= 1ull << (f1 + 1);
            }
        }
    } else {
        if (type == BISHOP || type == QUEEN) cand |= rays(sq, occ, true);
        if (type == ROOK || type == QUEEN) cand |= rays(sq, occ, false);
    }
    cand &= ~own;
    if (my_king == 0ull) return cand | (ep_target & ~own);  // no king to protect
    // a piece that shields the king from a slider moves only along the shielding line
    const bool pinned = first_on_ray && (beyond & (ray_diag ? e.diag : e.line)) != 0ull;
    unsigned long long legal = cand & target_mask & (pinned ? line : ~0ull);
    // en passant takes two pieces off one rank at once: tested on the position after the move
    for (unsigned long long rest = ep_target & ~own; rest != 0ull; rest &= rest - 1ull) {
        const int t = __ffsll(static_cast<long long>(rest)) - 1;
        const unsigned long long tb = 1ull << t;
        const unsigned long long gone = 1ull << (t - (black ? -8 : 8));
        const unsigned long long after = ((occ & ~bb) & ~gone) | tb;
        if (!attacked(king_sq, after, without(e, gone))) legal |= tb;
    }
    return legal;
}

// ------------------------------------------------------------------------------------------
// One THREAD per board: the stand-alone generator for launches that fill the GPU.  A board is 64
// bytes; with a warp per board every bitboard costs warp-wide reductions over 32 lanes that hold
// one piece each.  A thread that keeps the whole board needs none, and only the mover's own pieces
// are visited one by one; slot p has the same piece type on almost every board (promotions aside),
// so the threads of a warp take the same branch as they walk the slots.  Boards come in and legal
// words go out through shared memory so that global accesses stay coalesced.
// ------------------------------------------------------------------------------------------
template <int kShift>
__device__ __forceinline__ unsigned long long fill_ray(unsigned long long gen, unsigned long long occ,
                                                       unsigned long long wrap) {
    // the pieces' bits spread over empty squares in doubling steps (1, 2, 4), then one more
    // step lands on the first occupied square; `wrap` clears the file a step must not arrive on
    unsigned long long pro = ~occ & wrap;
    if constexpr (kShift > 0) {
        gen |= pro & (gen << kShift);
        pro &= pro << kShift;
        gen |= pro & (gen << (2 * kShift));
        pro &= pro << (2 * kShift);
        gen |= pro & (gen << (4 * kShift));
        return (gen << kShift) & wrap;
    } else {
        gen |= pro & (gen >> -kShift);
        pro &= pro >> -kShift;
        gen |= pro & (gen >> (-2 * kShift));
        pro &= pro >> (-2 * kShift);
        gen |= pro & (gen >> (-4 * kShift));
        return (gen >> -kShift) & wrap;
    }
}
// Squares seen from every piece of the set `b` along the bishop or the rook lines.
__device__ __forceinline__ unsigned long long fill_diag(unsigned long long b, unsigned long long occ) {
    return fill_ray<9>(b, occ, ~kFileA) | fill_ray<7>(b, occ, ~kFileH) | fill_ray<-7>(b, occ, ~kFileA) |
           fill_ray<-9>(b, occ, ~kFileH);
}
__device__ __forceinline__ unsigned long long fill_line(unsigned long long b, unsigned long long occ) {
    return fill_ray<8>(b, occ, ~0ull) | fill_ray<-8>(b, occ, ~0ull) | fill_ray<1>(b, occ, ~kFileA) |
           fill_ray<-1>(b, occ, ~kFileH);
}
// Squares a set of pawns of one colour attacks.
__device__ __forceinline__ unsigned long long pawn_attacks(unsigned long long b, bool black_pawns) {
    return black_pawns ? (((b >> 9) & ~kFileH) | ((b >> 7) & ~kFileA)) : (((b << 7) & ~kFileH) | ((b << 9) & ~kFileA));
}
// The whole rank, file or diagonal through two aligned squares (0 when they are not aligned).
__device__ __forceinline__ unsigned long long line_through(int a, int b) {
    const int ra = a >> 3, fa = a & 7, rb = b >> 3, fb = b & 7;
    if (ra == rb) return 0xFFull << (8 * ra);
    if (fa == fb) return kFileA << fa;
    if (ra - fa == rb - fb) {
        const int d = ra - fa;                                   // the a1-h8 diagonal moved up or down
        return d >= 0 ? 0x8040201008040201ull << (8 * d) : 0x8040201008040201ull >> (-8 * d);
    }
    if (ra + fa == rb + fb) {
        const int d = ra + fa - 7;                               // the h1-a8 diagonal moved up or down
        return d >= 0 ? 0x0102040810204080ull << (8 * d) : 0x0102040810204080ull >> (-8 * d);
    }
    return 0ull;
}

constexpr int kTpbThreads = 128;
constexpr int kTpbInStride = 17;      // 32-bit words per board in shared memory (16 + 1: no bank conflicts)
constexpr int kTpbOutStride = 17;     // 64-bit words per board in shared memory: the mover's (16 + 1)
constexpr int kTpbMaskStride = 33;    // a random ply's incoming words (32 + 1)

__device__ __forceinline__ unsigned piece_word(const unsigned* my, int p) {
    return (my[p >> 1] >> (16 * (p & 1))) & 0xFFFFu;
}
// x << s of a 64-bit word with a single bit at 0, 0 for s >= 64 (32-bit shifts clamp).
__device__ __forceinline__ unsigned long long bit_at(unsigned s) {
    unsigned lo, hi;
    asm("shl.b32 %0, 1, %1;" : "=r"(lo) : "r"(s));
    asm("shl.b32 %0, 1, %1;" : "=r"(hi) : "r"(s - 32u));
    return (static_cast<unsigned long long>(hi) << 32) | lo;
}
// The legal words of one board held by one thread: `my` = the board's 32 piece words as 16
// 32-bit words, `out[0..31]` receives the legal-target word of every slot.  Returns whether the
// side to move is in check.  This form takes any board; `board_moves` below is the faster one for boards
// whose pieces are in the slots they start in.
//
// A board with black to move is turned upside down as it is decoded (and its words on the way out), so that
// nothing below depends on the side to move; the bitboards are bit planes of the words, without a branch per
// piece; checks and pins are taken ray by ray from the king without loops.
__device__ __noinline__ bool board_moves_any(const unsigned* my, bool black, unsigned long long* out) {
    // ---- pass 1: bit planes.  A captured piece's square is moved off the board ----
    const unsigned flip = black ? 0x00380038u : 0u;
    unsigned long long half[2] = {0ull, 0ull}, t0 = 0, t1 = 0, t2 = 0, sp = 0;
    unsigned stray = 0u;                 // a live piece whose colour is not its slot's (white 0-15, black 16-31)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll 4
        for (int q = 0; q < 8; ++q) {
            const unsigned two = my[8 * h + q] ^ flip;
            stray |= (two ^ (h ? 0x04000400u : 0u)) & ~(two >> 1);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const unsigned w = k ? two >> 16 : two;
                const unsigned long long bb = bit_at((w & 63u) | ((w >> 5) & 64u));
                half[h] |= bb;
                t0 |= (w & 0x040u) ? bb : 0ull;
                t1 |= (w & 0x080u) ? bb : 0ull;
                t2 |= (w & 0x100u) ? bb : 0ull;
                sp |= (w & 0x200u) ? bb : 0ull;
            }
        }
    const bool by_slot = (stray & 0x04000400u) == 0u;
    const unsigned long long occ = half[0] | half[1];
    unsigned long long own = black ? half[1] : half[0];
    if (!by_slot) {
        own = 0ull;
#pragma unroll 1
        for (int p = 0; p < 32; ++p) {
            const unsigned w = piece_word(my, p) ^ (flip & 63u);
            if (((w & 0x400u) != 0u) == black) own |= bit_at((w & 63u) | ((w >> 5) & 64u));
        }
    }
    const unsigned long long opp = occ & ~own, queens = t2 & ~(t1 | t0), pawns = occ & ~(t0 | t1 | t2);
    const unsigned long long kings = t2 & t0 & ~t1, rooks = t1 & t0 & ~t2;
    const unsigned long long e_pawns = opp & pawns, ep_pawns = e_pawns & sp, e_knights = opp & t0 & ~(t1 | t2);
    const unsigned long long e_diag = opp & ((t1 & ~(t0 | t2)) | queens), e_line = opp & (rooks | queens);
    const unsigned long long e_king = opp & kings, my_king = own & kings, fresh_rooks = own & rooks & ~sp;
    const int king_sq = my_king ? __ffsll(static_cast<long long>(my_king)) - 1 : 0;
    // ---- what the opponent attacks, with the mover's king lifted off the board ----
    const unsigned long long occ_nk = occ & ~my_king;
    const unsigned long long danger = pawn_attacks(e_pawns, true) | knight_pattern(e_knights) |
                                      king_pattern(e_king) | fill_diag(e_diag, occ_nk) | fill_line(e_line, occ_nk);
    // ---- the eight rays from the king: is the first piece a checker (the squares up to it answer the
    //      check), or an own piece with a slider of the ray's kind next behind it ----
    const unsigned long long kd_ex = diag_ex(king_sq), ka_ex = anti_ex(king_sq), kr_ex = rank_ex(king_sq),
                             kf_ex = file_ex(king_sq);
    const unsigned long long above = 0ull - (my_king << 1);          // squares above the king's
    const unsigned long long leapers = (knight_pattern(my_king) & e_knights) | (pawn_attacks(my_king, false) & e_pawns);
    unsigned long long answers = leapers, pinned = 0ull;
    int checkers = __popcll(leapers);
    auto line = [&](unsigned long long ex, unsigned long long sliders) {
        const unsigned long long seen = line_attacks(my_king, occ, ex), shields = seen & own;
        const unsigned long long next = line_attacks(my_king, occ & ~shields, ex) & ~seen & sliders, hit = seen & sliders;
        if (hit & above) { ++checkers; answers |= seen & above; }
        if (hit & ~above) { ++checkers; answers |= seen & ~above; }
        if (next & above) pinned |= shields & above;
        if (next & ~above) pinned |= shields & ~above;
    };
    line(kd_ex, e_diag);
    line(ka_ex, e_diag);
    line(kr_ex, e_line);
    line(kf_ex, e_line);
    const bool chk = checkers != 0;
    // one checker: the other pieces may only capture it or step between; two: only the king moves
    const unsigned long long target_mask = checkers == 0 ? ~0ull : (checkers == 1 ? answers : 0ull);
    // ---- the mover's pieces, one by one: its sixteen slots (all thirty-two for a board that
    //      does not keep the colours apart by slot) ----
    const int p_lo = by_slot ? (black ? 16 : 0) : 0, p_n = by_slot ? 16 : 32;
    const unsigned sel_lo = black ? 0x4567u : 0x3210u, sel_hi = black ? 0x0123u : 0x7654u;
    if (by_slot)
#pragma unroll 4
        for (int p = 0; p < 16; ++p) out[(p_lo ^ 16) + p] = 0ull;
#pragma unroll 1
    for (int i = 0; i < p_n; ++i) {
        const int p = p_lo + i;
        const unsigned word = piece_word(my, p) ^ (flip & 63u);
        unsigned long long legal = 0ull;
        if ((word & 0x800u) == 0u && ((word & 0x400u) != 0u) == black) {
            const bool special = (word & 0x200u) != 0u;
            const int type = (word >> 6) & 7, sq = word & 63;
            const unsigned long long bb = bit_at(sq);
            if (type == KING) {
                legal = king_pattern(bb) & ~danger;
                // castling: neither the king's square nor the one it crosses nor the one it lands on may
                // be attacked
                if (!special && !chk) {
                    if ((fresh_rooks & 0x80ull) && ((occ | danger) & 0x60ull) == 0ull) legal |= 0x40ull;
                    if ((fresh_rooks & 0x01ull) && (occ & 0x0Eull) == 0ull && (danger & 0x0Cull) == 0ull) legal |= 0x04ull;
                }
                legal &= ~own;
            } else {
                unsigned long long cand = 0ull, ep = 0ull;
                if (type == PAWN) {
                    const unsigned long long one = (bb << 8) & ~occ, att = pawn_attacks(bb, false);
                    const unsigned long long two = (sq >> 3) == 1 ? (one << 8) & ~occ : 0ull;
                    cand = one | two | (att & opp);
                    // en passant: an enemy pawn that has just made its double step stands beside us
                    if ((sq >> 3) == 4) ep = att & (ep_pawns << 8) & ~own;
                } else if (type == KNIGHT) {
                    cand = knight_pattern(bb);
                } else {
                    if (type == BISHOP || type == QUEEN)
                        cand |= line_attacks(bb, occ, diag_ex(sq)) | line_attacks(bb, occ, anti_ex(sq));
                    if (type == ROOK || type == QUEEN)
                        cand |= line_attacks(bb, occ, rank_ex(sq)) | line_attacks(bb, occ, file_ex(sq));
                }
                legal = cand & ~own & target_mask;
                // a piece that shields the king from a slider moves only along that line
                if (bb & pinned) legal &= (bb & kd_ex) ? kd_ex : (bb & ka_ex) ? ka_ex : (bb & kr_ex) ? kr_ex : kf_ex;
                // en passant takes two pieces off one rank at once: tested on the position after it
                for (; ep != 0ull; ep &= ep - 1ull) {
                    const unsigned long long tb = ep & (0ull - ep), gone = tb >> 8;
                    const unsigned long long after = ((occ & ~bb) & ~gone) | tb;
                    const bool hit = (knight_pattern(my_king) & e_knights) != 0ull ||
                                     (pawn_attacks(my_king, false) & (e_pawns & ~gone)) != 0ull ||
                                     (king_pattern(my_king) & e_king) != 0ull ||
                                     ((line_attacks(my_king, after, kd_ex) | line_attacks(my_king, after, ka_ex)) & e_diag) != 0ull ||
                                     ((line_attacks(my_king, after, kr_ex) | line_attacks(my_king, after, kf_ex)) & e_line) != 0ull;
                    if (!hit) legal |= tb;
                }
            }
        }
        const unsigned lo = static_cast<unsigned>(legal), hi = static_cast<unsigned>(legal >> 32);
        out[p] = (static_cast<unsigned long long>(__byte_perm(lo, hi, sel_hi)) << 32) | __byte_perm(lo, hi, sel_lo);
    }
    return chk;
}

// ---- the faster form of the same, for boards whose pieces are in the slots they start in ----
// What a slider sees along one line, looked up: the line's squares are folded into one byte (a rank, a
// diagonal and an antidiagonal hold one square of each file, so the fold is two logical operations and a
// multiplication), whose inner six bits pick the answer for the slider's file.  A file is folded by rank.  (The method is
// published as kindergarten bitboards.)
// Row 64 of the tables by square, and rank 8 of `up`, are empty: a captured piece looks there.
struct alignas(16) MoveTables {
    unsigned long long up[9 * 64];               // [rank][ranks 2-7 occupied]: squares of the a file
    unsigned long long diag[65][2];              // both diagonals through a square, the square included
    unsigned along[8 * 64];                      // [file][files b-g occupied]: a byte of files, four times
    unsigned long long rank[65], knight[65], king[65], pawn[65];   // pawn: what a white pawn attacks
    unsigned long long pad[1];
};
constexpr MoveTables make_move_tables() {
    MoveTables t{};
    for (int at = 0; at < 8; ++at)
        for (int inner = 0; inner < 64; ++inner) {
            const int occ = inner << 1;
            unsigned bits = 0;
            for (int i = at + 1; i < 8; ++i) { bits |= 1u << i; if ((occ >> i) & 1) break; }
            for (int i = at - 1; i >= 0; --i) { bits |= 1u << i; if ((occ >> i) & 1) break; }
            t.along[at * 64 + inner] = bits * 0x01010101u;
            for (int i = 0; i < 8; ++i)
                if ((bits >> i) & 1u) t.up[at * 64 + inner] |= 1ull << (8 * i);
        }
    for (int sq = 0; sq < 64; ++sq)
        for (int to = 0; to < 64; ++to) {
            const int dr = (to >> 3) - (sq >> 3), df = (to & 7) - (sq & 7);
            const int r = dr < 0 ? -dr : dr, f = df < 0 ? -df : df;
            const unsigned long long b = 1ull << to;
            if (dr == df) t.diag[sq][0] |= b;
            if (dr == -df) t.diag[sq][1] |= b;
            if (dr == 0) t.rank[sq] |= b;
            if ((r == 1 && f == 2) || (r == 2 && f == 1)) t.knight[sq] |= b;
            if (r <= 1 && f <= 1 && r + f > 0) t.king[sq] |= b;
            if (dr == 1 && f == 1) t.pawn[sq] |= b;
        }
    return t;
}
__device__ const MoveTables kMoveTables = make_move_tables();

// Along a rank or a diagonal (`line`, which holds the slider's square) from a square of file sq & 7.
__device__ __forceinline__ unsigned long long see_along(const MoveTables& t, unsigned long long occ, unsigned long long line,
                                                        unsigned sq) {
    const unsigned long long o = occ & line;
    const unsigned fold = static_cast<unsigned>(o) | static_cast<unsigned>(o >> 32);
    const unsigned f = t.along[(sq & 7u) * 64u + (fold * 0x02020202u >> 26)];
    return line & ((static_cast<unsigned long long>(f) << 32) | f);
}
// Along the file of a square (64: nothing).
__device__ __forceinline__ unsigned long long see_file(const MoveTables& t, unsigned long long occ, unsigned sq) {
    const unsigned f = sq & 7u;
    const unsigned lo = (static_cast<unsigned>(occ) >> f) & 0x01010101u, hi = (static_cast<unsigned>(occ >> 32) >> f) & 0x01010101u;
    const unsigned long long u = t.up[(sq >> 3) * 64u + ((hi * 16u + lo) * 0x02040810u >> 26)];
    return (static_cast<unsigned long long>(static_cast<unsigned>(u >> 32) << f) << 32) | (static_cast<unsigned>(u) << f);
}
__device__ __forceinline__ unsigned long long see_diag(const MoveTables& t, unsigned long long occ, unsigned sq) {
    const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(t.diag[sq]);
    return see_along(t, occ, d.x, sq) | see_along(t, occ, d.y, sq);
}
__device__ __forceinline__ unsigned long long see_line(const MoveTables& t, unsigned long long occ, unsigned sq) {
    return see_along(t, occ, t.rank[sq], sq) | see_file(t, occ, sq);
}

// A piece word with its slot's expected colour and type taken out: its square when the piece is there, 64
// or more when it has been captured or is not the piece expected, so that `bit_at` of it is its bit or 0.
constexpr unsigned kIndexBits = 0x0DFF0DFFu;

// The legal words of one board held by one thread: the mover's sixteen into `to`, the other side's are
// zero -- or, where the board takes the general form, all thirty-two into `all`, and `by_slot` is false.
//
// A colour's sixteen slots are eight pawns, two knights, two bishops, two rooks, the queen and the king,
// and only pawns ever change their type.  So a piece's plane is known before its word is looked at, its
// bit falls out of the word and the expectation in five operations, and each slot has code of its own, with no
// branch on what it holds.  Promoted pawns (one board in thirty of random games) are found by
// counting: the planes must hold as many squares as there are pieces left.  They are put in one by one; a board
// that does not add up then (colours or types in other slots, two pieces on a square) takes the general form.
//
// Bound by the integer pipe (the general form keeps it busy 87 % of the time with 3,600 instructions a board), which is why
// every attack is a table's.  The loops over the pawns stay loops: unrolled, the code misses the instruction cache (107 us).
// 2^20 boards of random games, B200: 102 us, 161 in the general form (323 bytes a board: 3.3 and 2.1 TB/s of the 6.5 a
// copy reaches); 2,400 instructions a board, the integer pipe 76 % busy.
__device__ __forceinline__ bool board_moves(const unsigned* my, bool black, unsigned long long* to, unsigned long long* all,
                                            const MoveTables& t, bool& by_slot) {
    by_slot = true;
    const unsigned flip = black ? 0x04380438u : 0u;             // the mover is white: squares turned, colour changed
    const unsigned* mine = my + (black ? 8 : 0);
    const unsigned* theirs = my + (black ? 0 : 8);
    constexpr unsigned kTheirs = 0x04000400u, kN = 0x00400040u, kB = 0x00800080u, kR = 0x00C000C0u, kQK = 0x01400100u;
    auto lo_of = [](unsigned x) { return x & 0xFFFFu; };
    auto hi_of = [](unsigned x) { return x >> 16; };
    auto expect = [&](unsigned two, unsigned e) { return (two ^ (flip ^ e)) & kIndexBits; };
    auto both = [&](unsigned x) { return bit_at(lo_of(x)) | bit_at(hi_of(x)); };
    auto on_board = [](unsigned i) { return min(i, 64u); };
    // ---- the planes ----
    unsigned long long own_pawns = 0ull, e_pawns = 0ull;
    unsigned gone = 0u, stepped = 0u;                            // captured pieces, counted; enemy pawns that are flagged
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const unsigned a = mine[q], b = theirs[q];
        own_pawns |= both(expect(a, 0u));
        e_pawns |= both(expect(b, kTheirs));
        gone += (a & 0x08000800u) + (b & 0x08000800u);
        stepped |= b & 0x02000200u;
    }
    const unsigned w_n = mine[4], w_b = mine[5], w_r = mine[6], w_qk = mine[7];
    const unsigned v_n = theirs[4], v_b = theirs[5], v_r = theirs[6], v_qk = theirs[7];
    gone += (w_n & 0x08000800u) + (w_b & 0x08000800u) + (w_r & 0x08000800u) + (w_qk & 0x08000800u);
    gone += (v_n & 0x08000800u) + (v_b & 0x08000800u) + (v_r & 0x08000800u) + (v_qk & 0x08000800u);
    const unsigned x_qk = expect(w_qk, kQK), y_n = expect(v_n, kTheirs | kN), y_b = expect(v_b, kTheirs | kB),
                   y_r = expect(v_r, kTheirs | kR), y_qk = expect(v_qk, kTheirs | kQK);
    const unsigned long long my_king = bit_at(hi_of(x_qk)), e_king = bit_at(hi_of(y_qk)), e_queen = bit_at(lo_of(y_qk));
    unsigned long long e_knights = both(y_n), e_diag = both(y_b) | e_queen, e_line = both(y_r) | e_queen;
    unsigned long long own = own_pawns | both(expect(w_n, kN)) | both(expect(w_b, kB)) | both(expect(w_r, kR)) |
                             bit_at(lo_of(x_qk)) | my_king;
    unsigned long long occ = own | e_pawns | e_knights | e_diag | e_line | e_king;
    // castling rooks: not moved, on their corners
    const unsigned r_lo = lo_of(w_r ^ flip ^ kR) & 0xFFFu, r_hi = hi_of(w_r ^ flip ^ kR) & 0xFFFu;
    bool fresh_a = r_lo == 0u || r_hi == 0u, fresh_h = r_lo == 7u || r_hi == 7u;
    const int live = 32 - static_cast<int>((gone & 0xFFFFu) >> 11) - static_cast<int>(gone >> 27);
    // ---- promoted pawns ----
    unsigned own_promoted = 0u;                                  // the mover's, by slot
    unsigned long long e_promoted = 0ull;                        // the opponent's sliders
    if (__popcll(occ) != live) {
        unsigned todo = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned a = (mine[q] & 0x01C001C0u) + 0x01C001C0u, b = (theirs[q] & 0x01C001C0u) + 0x01C001C0u;
            todo |= ((a & 0x02000200u) >> (9 - q)) | ((b & 0x02000200u) >> (5 - q));
        }
        for (; todo != 0u; todo &= todo - 1u) {
            const int i = __ffs(static_cast<int>(todo)) - 1, q = i & 3;
            const bool enemy = (i & 4) != 0;
            const unsigned word = ((enemy ? theirs : mine)[q] >> (i & 16)) ^ (flip & 0x438u);
            const int type = (word >> 6) & 7;
            if ((word & 0x800u) != 0u || ((word & 0x400u) != 0u) != enemy || type < KNIGHT || type > QUEEN) continue;
            const unsigned long long bb = bit_at(word & 63u);
            occ |= bb;
            if (enemy) {
                if (type == KNIGHT) e_knights |= bb;
                if (type == BISHOP || type == QUEEN) e_diag |= bb;
                if (type == ROOK || type == QUEEN) e_line |= bb;
                if (type != KNIGHT) e_promoted |= bb;
            } else {
                own |= bb;
                own_promoted |= 1u << (2 * q + (i >> 4));
                if (type == ROOK && (word & 0x200u) == 0u) { fresh_a |= (word & 63u) == 0u; fresh_h |= (word & 63u) == 7u; }
            }
        }
        by_slot = __popcll(occ) == live;
        if (!by_slot) return board_moves_any(my, black, all);
    }
    const unsigned long long opp = occ & ~own;
    // ---- what the opponent attacks, with the mover's king lifted off the board ----
    const unsigned long long occ_nk = occ & ~my_king;
    unsigned long long danger = pawn_attacks(e_pawns, true) | knight_pattern(e_knights) | t.king[on_board(hi_of(y_qk))];
    {
        const unsigned b0 = on_board(lo_of(y_b)), b1 = on_board(hi_of(y_b)), r0 = on_board(lo_of(y_r)), r1 = on_board(hi_of(y_r)),
                       qq = on_board(lo_of(y_qk));
        danger |= see_diag(t, occ_nk, b0) | see_diag(t, occ_nk, b1) | see_diag(t, occ_nk, qq);
        danger |= see_line(t, occ_nk, r0) | see_line(t, occ_nk, r1) | see_line(t, occ_nk, qq);
        for (; e_promoted != 0ull; e_promoted &= e_promoted - 1ull) {
            const unsigned sq = static_cast<unsigned>(__ffsll(static_cast<long long>(e_promoted)) - 1);
            const unsigned long long bb = e_promoted & (0ull - e_promoted);
            if (bb & e_diag) danger |= see_diag(t, occ_nk, sq);
            if (bb & e_line) danger |= see_line(t, occ_nk, sq);
        }
    }
    // ---- the four lines through the king: is the first piece on either side a checker (the squares up to it answer the
    //      check), or an own piece with a slider of the line's kind next behind it ----
    const unsigned ks = on_board(hi_of(x_qk));
    const unsigned long long above = 0ull - (my_king << 1);          // squares above the king's
    const ulonglong2 k_diag = *reinterpret_cast<const ulonglong2*>(t.diag[ks]);
    const unsigned long long k_rank = t.rank[ks], k_file = kFileA << (ks & 7u);
    const unsigned long long leapers = (t.knight[ks] & e_knights) | (t.pawn[ks] & e_pawns);
    unsigned long long answers = 0ull, pinned = 0ull, hits = 0ull;
    auto line = [&](unsigned long long sliders, auto&& see) {
        const unsigned long long seen = see(occ), shields = seen & own, hit = seen & sliders;
        const unsigned long long next = see(occ & ~shields) & ~seen & sliders;
        hits |= hit;
        if (hit != 0ull) answers |= seen;
        if (next & above) pinned |= shields & above;
        if (next & ~above) pinned |= shields & ~above;
    };
    line(e_diag, [&](unsigned long long o) { return see_along(t, o, k_diag.x, ks); });
    line(e_diag, [&](unsigned long long o) { return see_along(t, o, k_diag.y, ks); });
    line(e_line, [&](unsigned long long o) { return see_along(t, o, k_rank, ks); });
    line(e_line, [&](unsigned long long o) { return see_file(t, o, ks); });
    const int checkers = __popcll(hits) + __popcll(leapers);
    const bool chk = checkers != 0;
    // one checker: the other pieces may only capture it or step between; two: only the king moves
    const unsigned long long target_mask = checkers == 0 ? ~0ull
                                           : checkers == 1 ? leapers | (answers & ((hits & above) ? above : ~above)) : 0ull;
    // ---- the mover's pieces ----
    const unsigned long long allowed = target_mask & ~own;
    const unsigned sel_lo = black ? 0x4567u : 0x3210u, sel_hi = black ? 0x0123u : 0x7654u;
    auto put = [&](int slot, unsigned long long legal) {
        const unsigned lo = static_cast<unsigned>(legal), hi = static_cast<unsigned>(legal >> 32);
        to[slot] = (static_cast<unsigned long long>(__byte_perm(lo, hi, sel_hi)) << 32) | __byte_perm(lo, hi, sel_lo);
    };
    // a piece that shields the king from a slider moves only along that line
    auto held = [&](unsigned long long bb, unsigned long long legal) {
        if (bb & pinned)
            legal &= (bb & k_diag.x) ? k_diag.x : (bb & k_diag.y) ? k_diag.y : (bb & k_rank) ? k_rank : k_file;
        return legal;
    };
    {
        const unsigned long long step = ~occ & target_mask, takes = opp & target_mask;
        const unsigned long long two = ~occ & (~occ << 8) & target_mask & 0xFF000000ull;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            const unsigned x = expect(mine[q], 0u);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const unsigned i = k ? hi_of(x) : lo_of(x);
                const unsigned long long bb = bit_at(i);
                put(2 * q + k, held(bb, ((bb << 8) & step) | ((bb << 16) & two) | (t.pawn[on_board(i)] & takes)));
            }
        }
    }
    {
        const unsigned x_n = expect(w_n, kN), x_b = expect(w_b, kB), x_r = expect(w_r, kR);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned i = k ? hi_of(x_n) : lo_of(x_n);
            put(8 + k, held(bit_at(i), t.knight[on_board(i)] & allowed));
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned i = k ? hi_of(x_b) : lo_of(x_b);
            put(10 + k, held(bit_at(i), see_diag(t, occ, on_board(i)) & allowed));
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned i = k ? hi_of(x_r) : lo_of(x_r);
            put(12 + k, held(bit_at(i), see_line(t, occ, on_board(i)) & allowed));
        }
        const unsigned i = lo_of(x_qk);
        put(14, held(bit_at(i), (see_diag(t, occ, on_board(i)) | see_line(t, occ, on_board(i))) & allowed));
    }
    {
        unsigned long long legal = t.king[ks] & ~danger;
        // castling: neither the king's square nor the one it crosses nor the one it lands on may be attacked
        if (my_king != 0ull && (w_qk & 0x02000000u) == 0u && !chk) {
            if (fresh_h && ((occ | danger) & 0x60ull) == 0ull) legal |= 0x40ull;
            if (fresh_a && (occ & 0x0Eull) == 0ull && (danger & 0x0Cull) == 0ull) legal |= 0x04ull;
        }
        put(15, legal & ~own);
    }
    // ---- the mover's promoted pawns ----
    for (; own_promoted != 0u; own_promoted &= own_promoted - 1u) {
        const int slot = __ffs(static_cast<int>(own_promoted)) - 1;
        const unsigned word = (mine[slot >> 1] >> (16 * (slot & 1))) ^ (flip & 63u), sq = word & 63u;
        const int type = (word >> 6) & 7;
        unsigned long long cand = 0ull;
        if (type == KNIGHT) cand = t.knight[sq];
        if (type == BISHOP || type == QUEEN) cand |= see_diag(t, occ, sq);
        if (type == ROOK || type == QUEEN) cand |= see_line(t, occ, sq);
        put(slot, held(bit_at(sq), cand & allowed));
    }
    // ---- en passant takes two pieces off one rank at once: tested on the position after it ----
    if (stepped != 0u) {
        unsigned long long targets = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned b = theirs[q], x = expect(b, kTheirs);
            if (b & 0x0200u) targets |= bit_at(lo_of(x)) << 8;
            if (b & 0x02000000u) targets |= bit_at(hi_of(x)) << 8;
        }
        targets &= ~own & 0x0000FF0000000000ull;
        if (pawn_attacks(targets, true) & own_pawns)
#pragma unroll 1
            for (int slot = 0; slot < 8; ++slot) {
                const unsigned x = expect(mine[slot >> 1], 0u), i = (slot & 1) ? hi_of(x) : lo_of(x);
                const unsigned long long bb = bit_at(i);
                unsigned long long legal = 0ull;
                for (unsigned long long ep = t.pawn[on_board(i)] & targets; ep != 0ull; ep &= ep - 1ull) {
                    const unsigned long long tb = ep & (0ull - ep), victim = tb >> 8;
                    const unsigned long long after = ((occ & ~bb) & ~victim) | tb;
                    const bool hit = (t.knight[ks] & e_knights) != 0ull || (t.pawn[ks] & (e_pawns & ~victim)) != 0ull ||
                                     (t.king[ks] & e_king) != 0ull ||
                                     (see_diag(t, after, ks) & e_diag) != 0ull || (see_line(t, after, ks) & e_line) != 0ull;
                    if (!hit) legal |= tb;
                }
                const unsigned lo = static_cast<unsigned>(legal), hi = static_cast<unsigned>(legal >> 32);
                to[slot] |= (static_cast<unsigned long long>(__byte_perm(lo, hi, sel_hi)) << 32) | __byte_perm(lo, hi, sel_lo);
            }
    }
    return chk;
}

// Castling rights KQkq as four bits of a board held by one thread (torch_impl.py:294-318).
__device__ __forceinline__ unsigned board_rights(const unsigned* my) {
    bool wk = false, bk = false, k = false, q = false, k2 = false, q2 = false;
#pragma unroll 1
    for (int p = 0; p < 32; ++p) {
        const unsigned word = piece_word(my, p);
        if (((word >> 11) & 1u) || ((word >> 9) & 1u)) continue;
        const bool is_black = (word >> 10) & 1u;
        const int type = (word >> 6) & 7, sq = word & 63;
        if (type == KING) { if (is_black) bk = true; else wk = true; }
        if (type == ROOK) {
            if (!is_black) { k |= sq == 7; q |= sq == 0; }
            else { k2 |= sq == 63; q2 |= sq == 56; }
        }
    }
    return (wk && k ? 1u : 0u) | (wk && q ? 2u : 0u) | (bk && k2 ? 4u : 0u) | (bk && q2 ? 8u : 0u);
}
__device__ __forceinline__ void set_piece(unsigned* my, int p, unsigned v) {
    const int sh = 16 * (p & 1);
    my[p >> 1] = (my[p >> 1] & ~(0xFFFFu << sh)) | ((v & 0xFFFFu) << sh);
}
// Apply one move (`move` = slot * 64 + target, -1 = no move; `promo` 0..3 = N B R Q, negative =
// queen) to a board held by one thread: the reference's `step` without its hash
// (brokefish/env/torch_impl.py:412-548).  Capture: the first live piece on the target square, or
// for a pawn the en passant victim, which carries the double-step flag and stands beside the
// target's file neighbour, not on it.  `irreversible`: capture, pawn move or a change of
// castling rights.
__device__ __forceinline__ void board_step(unsigned* my, int control, int move, int promo, int& new_control,
                                           bool& irreversible) {
    new_control = control;
    irreversible = false;
    if (move < 0) return;
    const int source = move >> 6, target = move & 63;
    const bool white = control > 0;
    const unsigned mover = piece_word(my, source);
    const int mtype = (mover >> 6) & 7, from = mover & 63;
    const bool is_pawn = mtype == PAWN;
    const unsigned rights_before = board_rights(my);
    const unsigned victim_word = ((white ? 3u : 1u) << 9) + static_cast<unsigned>(target + (white ? -8 : 8));
    const int dx = target - from;
    const bool castling = mtype == KING && (dx == 2 || dx == -2);
    const int corner = (white ? 0 : 56) + (dx > 0 ? 7 : 0);
    int captured = -1, rook = -1;
#pragma unroll 1
    for (int p = 0; p < 32; ++p) {
        const unsigned word = piece_word(my, p);
        const bool live = ((word >> 11) & 1u) == 0u;
        if (captured < 0 && ((live && static_cast<int>(word & 63u) == target) || (is_pawn && word == victim_word)))
            captured = p;
    }
    if (captured >= 0) set_piece(my, captured, 1u << 11);
    // the corner rook is looked for by its square before anything moved, by its type after the capture
    if (castling) {
#pragma unroll 1
        for (int p = 0; p < 32; ++p) {
            const unsigned word = piece_word(my, p);
            const unsigned square = p == captured ? static_cast<unsigned>(target) : (word & 63u);
            if (rook < 0 && ((word >> 6) & 7u) == ROOK && static_cast<int>(square) == corner) rook = p;
        }
    }
    {
        unsigned w = (piece_word(my, source) & ~63u & 0xFFFu) + static_cast<unsigned>(target);
        if (is_pawn && (target >> 3) == (white ? 7 : 0))
            w += static_cast<unsigned>(promo < 0 ? QUEEN : promo + KNIGHT) << 6;
        if (mtype == KING || mtype == ROOK) w |= 1u << 9;
        set_piece(my, source, w);
    }
    if (rook >= 0)
        set_piece(my, rook, (piece_word(my, rook) & ~63u & 0xFFFu) + static_cast<unsigned>((white ? 0 : 56) + (dx > 0 ? 5 : 3)));
    // the en passant flag lives for one ply: clear every pawn's, set the double-stepper's
#pragma unroll 1
    for (int p = 0; p < 32; ++p) {
        const unsigned word = piece_word(my, p);
        if (((word >> 6) & 7u) == PAWN && ((word >> 9) & 1u)) set_piece(my, p, word & ~(1u << 9) & 0xFFFu);
    }
    if (is_pawn && (dx == 16 || dx == -16)) set_piece(my, source, piece_word(my, source) | (1u << 9));
    const int mag = (captured >= 0 || is_pawn) ? 1 : (control < 0 ? -control : control) + 1;
    new_control = white ? -mag : mag;
    irreversible = captured >= 0 || is_pawn || board_rights(my) != rights_before;
}

// Position keys.  The reference hashes a position with a table of random 64-bit keys indexed by
// (colour, type, square), side to move, the four castling rights and the file of a LEGAL en
// passant capture (brokefish/env/torch_impl.py:374-401, 321-371); only equality of hashes is
// ever used (repetition), so the keys here are this library's own: a 64-bit mix of the index.
__device__ __forceinline__ unsigned long long zobrist_key(int index) {
    unsigned long long x = 0x9E3779B97F4A7C15ull * static_cast<unsigned long long>(index + 1);
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
enum { ZOBRIST_SIDE = 768, ZOBRIST_CASTLE = 769, ZOBRIST_EP = 773 };

// Hash of a board held by one thread.  The en passant file counts only when a capture is really
// available: a pawn of the mover stands beside the pawn that has just made its double step, and
// taking it does not leave the mover's king attacked.
__device__ __forceinline__ unsigned long long board_hash(const unsigned* my, bool black) {
    unsigned long long h = black ? zobrist_key(ZOBRIST_SIDE) : 0ull;
    unsigned long long occ = 0, my_pawns = 0, my_king = 0, flagged = 0;
    unsigned long long e_pawns = 0, e_knights = 0, e_diag = 0, e_line = 0, e_king = 0;
#pragma unroll 1
    for (int p = 0; p < 32; ++p) {
        const unsigned word = piece_word(my, p);
        if ((word >> 11) & 1u) continue;
        const bool is_black = (word >> 10) & 1u, special = (word >> 9) & 1u;
        const int type = (word >> 6) & 7, sq = word & 63;
        const unsigned long long bb = 1ull << sq;
        h ^= zobrist_key(((is_black ? 6 : 0) + type) * 64 + sq);
        occ |= bb;
        if (is_black == black) {
            if (type == PAWN) my_pawns |= bb;
            if (type == KING) my_king |= bb;
        } else {
            if (type == PAWN) { e_pawns |= bb; if (special) flagged |= bb; }
            else if (type == KNIGHT) e_knights |= bb;
            else if (type == KING) e_king |= bb;
            else {
                if (type == BISHOP || type == QUEEN) e_diag |= bb;
                if (type == ROOK || type == QUEEN) e_line |= bb;
            }
        }
    }
    const unsigned rights = board_rights(my);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if ((rights >> i) & 1u) h ^= zobrist_key(ZOBRIST_CASTLE + i);
    if (flagged != 0ull) {
        const unsigned long long victim = flagged & (0ull - flagged);
        const int vsq = __ffsll(static_cast<long long>(victim)) - 1, vfile = vsq & 7;
        const unsigned long long target = black ? victim >> 8 : victim << 8;
        const int ksq = my_king ? __ffsll(static_cast<long long>(my_king)) - 1 : 0;
        bool legal = false;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const unsigned long long capturer = side ? ((victim << 1) & ~kFileA) : ((victim >> 1) & ~kFileH);
            if ((capturer & my_pawns) == 0ull) continue;
            const unsigned long long after = ((occ & ~capturer) & ~victim) | target;
            const bool hit = my_king != 0ull &&
                             ((knight_pattern(my_king) & e_knights) != 0ull ||
                              (pawn_attacks(my_king, black) & (e_pawns & ~victim)) != 0ull ||
                              (king_pattern(my_king) & e_king) != 0ull ||
                              ((line_attacks(my_king, after, diag_ex(ksq)) | line_attacks(my_king, after, anti_ex(ksq))) & e_diag) != 0ull ||
                              ((line_attacks(my_king, after, rank_ex(ksq)) | line_attacks(my_king, after, file_ex(ksq))) & e_line) != 0ull);
            legal |= !hit;
        }
        if (legal) h ^= zobrist_key(ZOBRIST_EP + vfile);
    }
    return h;
}

// Shared memory: the boards; the tables and the words that go out, or before them a random ply's incoming
// words.  (Launches without words need the boards only.)
constexpr int kTpbIn = kTpbThreads * kTpbInStride * 4;
constexpr int kTpbTables = static_cast<int>(sizeof(MoveTables));
constexpr int tpb_smem_bytes(bool pick, bool words) {
    const int made = kTpbTables + kTpbThreads * kTpbOutStride * 8, incoming = kTpbThreads * kTpbMaskStride * 8;
    return kTpbIn + (!words ? 0 : pick && incoming > made ? incoming : made);
}
static_assert(kTpbIn % 16 == 0 && kTpbTables % 16 == 0 && tpb_smem_bytes(true, true) <= 49152, "shared memory map");
// What becomes of a board's words: the first two are the side to move, whose words lie in shared memory.
enum { WORDS_WHITE = 0, WORDS_BLACK = 1, WORDS_STORED = 2, WORDS_KEPT = 3 };

// One thread per board, boards and legal words staged through shared memory for coalescing.
// `hash_out` non-null: the position key of the resulting board.
// kStep: play `move` first (or, with kPick, the floor(r * count)-th legal move of the incoming
// `mask` in (slot, square) order; a board without legal moves stays as it is) and write the new
// board, control word and irreversible flag; `mask` non-null: the legal words of the resulting
// board follow.  In place (boards_out == boards) is safe: a block reads all its boards first.
// (Six blocks to an SM, at 80 registers: left to itself the compiler takes 122 to 128, which leaves four and costs 10 % of
// the words of 2^20 boards, 20 % of a move without them.  With five a random ply is the faster.)
template <bool kStep, bool kPick>
__global__ void __launch_bounds__(kTpbThreads, kPick ? 5 : 6) engine_board_kernel(
        const uint16_t* boards, const int16_t* control, const int* move,
        const signed char* promo, const float* r, int n, uint16_t* boards_out,
        int16_t* control_out, unsigned char* irreversible, unsigned long long* mask,
        unsigned char* in_check, int* move_out, unsigned long long* hash_out) {
    extern __shared__ unsigned long long tpb_smem[];
    unsigned* s_in = reinterpret_cast<unsigned*>(tpb_smem);                                 // [128][17]
    MoveTables* s_tables = reinterpret_cast<MoveTables*>(reinterpret_cast<uint8_t*>(tpb_smem) + kTpbIn);
    unsigned long long* s_mask = reinterpret_cast<unsigned long long*>(s_tables);           // [128][33], before the tables
    unsigned long long* s_out = reinterpret_cast<unsigned long long*>(s_tables + 1);        // [128][17]
    const int tid = threadIdx.x;
    const long first = static_cast<long>(blockIdx.x) * kTpbThreads;
    const int here = static_cast<int>(min(static_cast<long>(kTpbThreads), n - first));
    // (every load is under way before the first is waited for: one after the other the tables' five alone are 1,500 cycles)
    constexpr int kTablePieces = (kTpbTables / 16 + kTpbThreads - 1) / kTpbThreads;
    uint4 piece[kTablePieces];
    auto load_tables = [&] {
#pragma unroll
        for (int k = 0; k < kTablePieces; ++k)
            if (tid + k * kTpbThreads < kTpbTables / 16)
                piece[k] = __ldg(reinterpret_cast<const uint4*>(&kMoveTables) + tid + k * kTpbThreads);
    };
    auto store_tables = [&] {
#pragma unroll
        for (int k = 0; k < kTablePieces; ++k)
            if (tid + k * kTpbThreads < kTpbTables / 16) reinterpret_cast<uint4*>(s_tables)[tid + k * kTpbThreads] = piece[k];
    };
    const bool tables = mask != nullptr;
    if (!kPick && tables) load_tables();
    after_previous_grid();
    {
        // coalesced load: the block's boards are one contiguous run of 16-byte pieces
        const uint4* src = reinterpret_cast<const uint4*>(boards + first * 32);
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (tid + k * kTpbThreads < here * 4) v[k] = src[tid + k * kTpbThreads];
        const int word = tid < here ? control[first + tid] : 1;
        if (kPick)
            for (int j = tid; j < here * 32; j += kTpbThreads)
                s_mask[(j >> 5) * kTpbMaskStride + (j & 31)] = mask[first * 32 + j];
        else if (tables)
            store_tables();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int j = tid + k * kTpbThreads;
            unsigned* d = s_in + (j >> 2) * kTpbInStride + (j & 3) * 4;
            if (j < here * 4) { d[0] = v[k].x; d[1] = v[k].y; d[2] = v[k].z; d[3] = v[k].w; }
        }
        s_in[tid * kTpbInStride + 16] = static_cast<unsigned>(word);      // (the row's padding)
    }
    __syncthreads();
    const bool mine = tid < here;
    unsigned* my = s_in + tid * kTpbInStride;
    int mv = -1;
    if (kPick) {
        if (mine) {
            const unsigned long long* words = s_mask + tid * kTpbMaskStride;
            int total = 0;
#pragma unroll 1
            for (int p = 0; p < 32; ++p) total += __popcll(words[p]);
            if (total > 0) {
                int pick = static_cast<int>(__fmul_rn(r[first + tid], static_cast<float>(total)));
                pick = pick < total - 1 ? pick : total - 1;
#pragma unroll 1
                for (int p = 0; p < 32 && mv < 0; ++p) {
                    unsigned long long m = words[p];
                    const int cnt = __popcll(m);
                    if (pick < cnt) {
                        for (int i = 0; i < pick; ++i) m &= m - 1ull;
                        mv = p * 64 + __ffsll(static_cast<long long>(m)) - 1;
                    }
                    pick -= cnt;
                }
            }
            if (move_out != nullptr) move_out[first + tid] = mv;
        }
        __syncthreads();                              // the incoming words' place is the tables'
        load_tables();
        store_tables();
        __syncthreads();
    }
    if (mine) {
        int ctl = static_cast<int>(my[16]);
        bool generate = mask != nullptr;
        if (kStep) {
            if (!kPick) mv = move[first + tid];
            if (kPick) generate = mv >= 0;            // a finished game keeps its (empty) legal words
            int nc;
            bool irr;
            board_step(my, ctl, mv, promo != nullptr ? promo[first + tid] : -1, nc, irr);
            if (!kPick || mv >= 0) {
                control_out[first + tid] = static_cast<int16_t>(nc);
                if (irreversible != nullptr) irreversible[first + tid] = irr ? 1 : 0;
            }
            ctl = nc;
        }
        unsigned words = WORDS_KEPT;
        if (generate) {
            bool by_slot;
            const bool chk = board_moves(my, ctl < 0, s_out + tid * kTpbOutStride, mask + (first + tid) * 32, *s_tables, by_slot);
            if (in_check != nullptr) in_check[first + tid] = chk ? 1 : 0;
            words = !by_slot ? WORDS_STORED : ctl < 0 ? WORDS_BLACK : WORDS_WHITE;
        }
        my[16] = words;
        if (hash_out != nullptr) hash_out[first + tid] = board_hash(my, ctl < 0);
    }
    if (!kStep) next_grid_may_start();
    __syncthreads();
    if (kStep) {
        // coalesced store of the block's boards (all of them: a board that did not move is rewritten as it was)
        uint4* dst = reinterpret_cast<uint4*>(boards_out + first * 32);
        for (int j = tid; j < here * 4; j += kTpbThreads) {
            const unsigned* d = s_in + (j >> 2) * kTpbInStride + (j & 3) * 4;
            dst[j] = make_uint4(d[0], d[1], d[2], d[3]);
        }
    }
    if (mask != nullptr) {
        // a warp stores a board's words; the side that is not to move has none
        const unsigned p = tid & 31, side = p >> 4;
#pragma unroll 4
        for (int b = tid >> 5; b < here; b += kTpbThreads / 32) {
            const unsigned words = s_in[b * kTpbInStride + 16];
            const unsigned long long v = s_out[b * kTpbOutStride + (p & 15)];
            if (words <= WORDS_BLACK) mask[(first + b) * 32 + p] = words == side ? v : 0ull;
        }
    }
}

// ------------------------------------------------------------------------------------------
// EIGHT LANES per board, four boards per warp: the form of a launch that does not fill the GPU.
// Lane j of a board holds slots j, 8 + j, 16 + j and 24 + j -- a white pawn, a white piece, a black
// pawn and a black piece on almost every board -- and direction j of the eight a slider moves along.
//
// A small launch is bound by the length of one thread's chain: a thread per board decodes 32 slots and
// then walks the mover's sixteen one after the other, 10 us for any number of boards up to 16,000 (29 us
// with a move before and a key after).  With eight lanes a lane decodes four words, the bitboards are
// completed by three xor-shuffles, the sliders' attacks are one fill with a different direction on every
// lane, so are the king's rays, and the mover's sixteen slots are two passes (pawns together, pieces
// together): 6 us (8 us) for 4096 boards.  It costs twice the thread form's instructions, so the large
// launches, bound by the integer pipe, keep that one.  Boards and legal words need no staging: a board's
// lanes read 16 contiguous bytes and write 64 at a time.
// ------------------------------------------------------------------------------------------
constexpr int kEngineThreads = 128;
constexpr int kEngineBoards = kEngineThreads / 8;       // boards per block

// ---- reductions over the eight lanes of a board (all 32 lanes of the warp take part) ----
__device__ __forceinline__ unsigned group_or(unsigned v) {
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) v |= __shfl_xor_sync(kFull, v, off);
    return v;
}
__device__ __forceinline__ unsigned long long group_or(unsigned long long v) {
    const unsigned lo = group_or(static_cast<unsigned>(v)), hi = group_or(static_cast<unsigned>(v >> 32));
    return (static_cast<unsigned long long>(hi) << 32) | lo;
}
__device__ __forceinline__ int group_min(int v) {
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) v = min(v, __shfl_xor_sync(kFull, v, off));
    return v;
}
__device__ __forceinline__ unsigned pick_word(const unsigned (&w)[4], int i) {
    const unsigned lo = (i & 1) ? w[1] : w[0], hi = (i & 1) ? w[3] : w[2];
    return (i & 2) ? hi : lo;
}
__device__ __forceinline__ void put_word(unsigned (&w)[4], int i, unsigned v) {
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = i == k ? v : w[k];
}

// A board as six bit planes over the squares: occupied, black, the three type bits, "special".
struct Board {
    unsigned long long occ, own;                 // own: the side to move's pieces
    unsigned long long e_pawns, e_knights, e_diag, e_line, e_king, ep_pawns;   // the opponent's; its
                                                 // pawns that have just made a double step
    unsigned long long my_king, my_pawns, fresh_rooks;
};
__device__ __forceinline__ Board board_planes(const unsigned (&w)[4], bool black) {
    unsigned long long occ = 0, blk = 0, t0 = 0, t1 = 0, t2 = 0, sp = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned word = w[i];
        const unsigned long long bb = static_cast<unsigned long long>((word >> 11 & 1u) ^ 1u) << (word & 63u);
        occ |= bb;
        if (word & 0x400u) blk |= bb;
        if (word & 0x040u) t0 |= bb;
        if (word & 0x080u) t1 |= bb;
        if (word & 0x100u) t2 |= bb;
        if (word & 0x200u) sp |= bb;
    }
    occ = group_or(occ); blk = group_or(blk); t0 = group_or(t0); t1 = group_or(t1); t2 = group_or(t2); sp = group_or(sp);
    Board b;
    b.occ = occ;
    b.own = black ? blk : occ & ~blk;
    const unsigned long long opp = occ & ~b.own;
    const unsigned long long pawns = occ & ~(t0 | t1 | t2), queens = t2 & ~(t1 | t0);
    b.e_pawns = opp & pawns;
    b.my_pawns = b.own & pawns;
    b.ep_pawns = b.e_pawns & sp;
    b.e_knights = opp & t0 & ~(t1 | t2);
    b.e_diag = opp & ((t1 & ~(t0 | t2)) | queens);
    b.e_line = opp & ((t1 & t0 & ~t2) | queens);
    const unsigned long long kings = t2 & t0 & ~t1;
    b.e_king = opp & kings;
    b.my_king = b.own & kings;
    b.fresh_rooks = b.own & t1 & t0 & ~(t2 | sp);
    return b;
}
// Is the mover's king attacked when the occupancy is `after` and the pawn `gone` has left?  (What
// an en passant capture, which takes two pieces off one rank at once, has to be tested with.)
__device__ __forceinline__ bool king_hit(const Board& b, bool black, unsigned long long after, unsigned long long gone) {
    if (b.my_king == 0ull) return false;
    const int sq = __ffsll(static_cast<long long>(b.my_king)) - 1;
    return (knight_pattern(b.my_king) & b.e_knights) != 0ull ||
           (pawn_attacks(b.my_king, black) & (b.e_pawns & ~gone)) != 0ull ||
           (king_pattern(b.my_king) & b.e_king) != 0ull ||
           ((line_attacks(b.my_king, after, diag_ex(sq)) | line_attacks(b.my_king, after, anti_ex(sq))) & b.e_diag) != 0ull ||
           ((line_attacks(b.my_king, after, rank_ex(sq)) | line_attacks(b.my_king, after, file_ex(sq))) & b.e_line) != 0ull;
}
// The set's bits spread over empty squares by `s` squares a step (doubling steps 1, 2, 4), then one
// more step lands on the first occupied square; `wrap` clears the file a step must not arrive on.
__device__ __forceinline__ unsigned long long fill_up(unsigned long long gen, unsigned long long occ, int s,
                                                      unsigned long long wrap) {
    unsigned long long pro = ~occ & wrap;
    gen |= pro & (gen << s);
    pro &= pro << s;
    gen |= pro & (gen << (2 * s));
    pro &= pro << (2 * s);
    gen |= pro & (gen << (4 * s));
    return (gen << s) & wrap;
}

// Legal words of the board into `mask` (the board's 32 words); returns whether the side to move is
// in check.  `store`: this board is to be written.
__device__ __forceinline__ bool group_moves(const unsigned (&w)[4], const Board& b, bool black, int lane, bool store,
                                            unsigned long long* mask) {
    const int j = lane & 7;
    const unsigned long long occ = b.occ, own = b.own, opp = occ & ~own, my_king = b.my_king;
    const int king_sq = my_king ? __ffsll(static_cast<long long>(my_king)) - 1 : 0;
    // ---- this lane's direction: up the board for lanes 0-3 (file, rank, the two diagonals), the
    //      same on the reversed board for lanes 4-7.  What the opponent's sliders attack along it
    //      with the mover's king lifted off the board; whether the first piece from the king is a
    //      checker; whether it is an own piece that shields the king from a slider behind it ----
    unsigned long long danger, answers, pinned;
    bool checks;
    {
        const int k = j & 3;
        const bool down = (j & 4) != 0;
        const int s = (0x7918 >> (4 * k)) & 15;
        const unsigned long long wrap = k == 0 ? ~0ull : (k == 3 ? ~kFileH : ~kFileA);
        auto flip = [&](unsigned long long v) { return down ? __brevll(v) : v; };
        const unsigned long long O = flip(occ), E = flip(k < 2 ? b.e_line : b.e_diag), K = flip(my_king), W = flip(own);
        danger = flip(fill_up(E, O & ~K, s, wrap));
        // the king's ray, and the ray from the first piece on it: on the whole line through the
        // king, subtracting a piece's bit from the occupancy flips the squares up to and including
        // the next occupied one
        const int ks = down ? 63 - king_sq : king_sq, kr = ks >> 3, kf = ks & 7;
        const int sh = k == 0 ? kf : 8 * (k == 1 ? kr : (k == 2 ? kr - kf : kr + kf - 7));
        const unsigned long long base = k == 0 ? kFileA : (k == 1 ? 0xFFull : (k == 2 ? 0x8040201008040201ull : 0x0102040810204080ull));
        const unsigned long long line = sh >= 0 ? base << sh : base >> -sh;
        const unsigned long long o1 = O & line & ~K, ray = (o1 ^ (o1 - K)) & line & ~K;
        checks = (ray & E) != 0ull;
        answers = checks ? flip(ray) : 0ull;
        const unsigned long long shield = ray & W, o2 = o1 & ~shield;
        pinned = ((o2 ^ (o2 - shield)) & line & ~shield & E) ? flip(shield) : 0ull;
    }
    danger = group_or(danger) | pawn_attacks(b.e_pawns, !black) | knight_pattern(b.e_knights) | king_pattern(b.e_king);
    answers = group_or(answers);
    pinned = group_or(pinned);
    const unsigned long long leapers = (knight_pattern(my_king) & b.e_knights) | (pawn_attacks(my_king, black) & b.e_pawns);
    const int checkers = __popc((__ballot_sync(kFull, checks) >> (lane & 24)) & 0xFFu) + __popcll(leapers);
    const bool chk = checkers != 0;
    // one checker: the other pieces may only capture it or step between; two: only the king moves
    const unsigned long long target_mask = checkers == 0 ? ~0ull : (checkers == 1 ? answers | leapers : 0ull);

    // ---- the mover's pieces: its pawn slots, then its piece slots; the other colour's slots only
    //      when some board of the warp does not keep the colours apart by slot ----
    bool mine[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) mine[i] = (w[i] & 0x800u) == 0u && ((w[i] & 0x400u) != 0u) == black;
    const bool stray = black ? (mine[0] || mine[1]) : (mine[2] || mine[3]);
    const int passes = __any_sync(kFull, stray) ? 4 : 2;
#pragma unroll 1
    for (int pass = 0; pass < passes; ++pass) {
        const int i = black ? pass ^ 2 : pass;
        const unsigned word = pick_word(w, i);
        unsigned long long legal = 0ull;
        if ((word & 0x800u) == 0u && ((word & 0x400u) != 0u) == black) {
            const bool special = (word & 0x200u) != 0u;
            const int type = (word >> 6) & 7, sq = word & 63;
            const unsigned long long bb = 1ull << sq;
            if (type == KING) {
                legal = king_pattern(bb) & ~danger;
                // castling: neither the king's square nor the one it crosses nor the one it lands on
                // may be attacked
                if (!special && !chk) {
                    const int row = black ? 56 : 0;
                    if ((b.fresh_rooks >> (row + 7)) & 1ull)
                        if (((occ >> (row + 5)) & 3ull) == 0ull && ((danger >> (row + 5)) & 3ull) == 0ull)
                            legal |= 1ull << (row + 6);
                    if ((b.fresh_rooks >> row) & 1ull)
                        if (((occ >> (row + 1)) & 7ull) == 0ull && ((danger >> (row + 2)) & 3ull) == 0ull)
                            legal |= 1ull << (row + 2);
                }
                legal &= ~own;
            } else {
                unsigned long long cand = 0ull, ep = 0ull;
                if (type == PAWN) {
                    const int rank = sq >> 3;
                    unsigned long long one, two;
                    if (black) {
                        one = (bb >> 8) & ~occ;
                        two = rank == 6 ? (one >> 8) & ~occ : 0ull;
                    } else {
                        one = (bb << 8) & ~occ;
                        two = rank == 1 ? (one << 8) & ~occ : 0ull;
                    }
                    const unsigned long long att = pawn_attacks(bb, black);
                    cand = one | two | (att & opp);
                    // en passant: an enemy pawn that has just made its double step stands beside us
                    if (b.ep_pawns != 0ull && rank == (black ? 3 : 4))
                        ep = att & (black ? b.ep_pawns >> 8 : b.ep_pawns << 8) & ~own;
                } else if (type == KNIGHT) {
                    cand = knight_pattern(bb);
                } else {
                    if (type == BISHOP || type == QUEEN)
                        cand |= line_attacks(bb, occ, diag_ex(sq)) | line_attacks(bb, occ, anti_ex(sq));
                    if (type == ROOK || type == QUEEN)
                        cand |= line_attacks(bb, occ, rank_ex(sq)) | line_attacks(bb, occ, file_ex(sq));
                }
                legal = cand & ~own & target_mask;
                if (bb & pinned) legal &= line_through(king_sq, sq);
                for (; ep != 0ull; ep &= ep - 1ull) {
                    const unsigned long long tb = ep & (0ull - ep);
                    const unsigned long long gone = black ? tb << 8 : tb >> 8;
                    if (!king_hit(b, black, ((occ & ~bb) & ~gone) | tb, gone)) legal |= tb;
                }
            }
        }
        if (store) mask[8 * i + j] = legal;
    }
    if (passes == 2 && store) {
        mask[(black ? 0 : 16) + j] = 0ull;
        mask[(black ? 8 : 24) + j] = 0ull;
    }
    return chk;
}

// Castling rights KQkq as four bits (torch_impl.py:294-318).
__device__ __forceinline__ unsigned group_rights(const unsigned (&w)[4]) {
    unsigned f = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned word = w[i];
        if (word & 0xA00u) continue;                                // captured, or has moved
        const bool is_black = (word & 0x400u) != 0u;
        const int type = (word >> 6) & 7, sq = word & 63;
        if (type == KING) f |= is_black ? 32u : 16u;
        if (type == ROOK) {
            if (!is_black) f |= (sq == 7 ? 1u : 0u) | (sq == 0 ? 2u : 0u);
            else           f |= (sq == 63 ? 4u : 0u) | (sq == 56 ? 8u : 0u);
        }
    }
    f = group_or(f);
    return ((f & 16u) ? f & 3u : 0u) | ((f & 32u) ? f & 12u : 0u);
}
// Apply one move (`move` = slot * 64 + target, -1 = no move; `promo` 0..3 = N B R Q, negative =
// queen): the reference's `step` without its hash (brokefish/env/torch_impl.py:412-548).  Capture:
// the first live piece on the target square, or for a pawn the en passant victim, which carries the
// double-step flag and stands beside the target's file neighbour, not on it.  `irreversible`:
// capture, pawn move or a change of castling rights.
__device__ __forceinline__ void group_step(unsigned (&w)[4], int lane, int control, int move, int promo, int& new_control,
                                           bool& irreversible) {
    const int j = lane & 7;
    const bool moves = move >= 0;
    const int source = moves ? (move >> 6) & 31 : 0, target = move & 63;
    const bool white = control > 0;
    const unsigned mover = __shfl_sync(kFull, pick_word(w, source >> 3), source & 7, 8);
    const int mtype = (mover >> 6) & 7, from = mover & 63;
    const bool is_pawn = mtype == PAWN;
    const unsigned rights_before = group_rights(w);
    const unsigned victim_word = ((white ? 3u : 1u) << 9) + static_cast<unsigned>(target + (white ? -8 : 8));
    const int dx = target - from;
    const bool castling = moves && mtype == KING && (dx == 2 || dx == -2);
    int captured = 32;
#pragma unroll
    for (int i = 3; i >= 0; --i)
        if (((w[i] & 0x800u) == 0u && static_cast<int>(w[i] & 63u) == target) || (is_pawn && w[i] == victim_word))
            captured = 8 * i + j;
    captured = group_min(captured);
    // the corner rook is looked for by its square before anything moved, by its type after the capture
    int rook = 32;
    if (__any_sync(kFull, castling)) {
        const int corner = (white ? 0 : 56) + (dx > 0 ? 7 : 0);
#pragma unroll
        for (int i = 3; i >= 0; --i)
            if (castling && 8 * i + j != captured && ((w[i] >> 6) & 7u) == ROOK && static_cast<int>(w[i] & 63u) == corner)
                rook = 8 * i + j;
        rook = group_min(rook);
    }
    if (moves) {
        if ((captured & 7) == j && captured < 32) put_word(w, captured >> 3, 1u << 11);
        if ((source & 7) == j) {
            unsigned v = (pick_word(w, source >> 3) & ~63u & 0xFFFu) + static_cast<unsigned>(target);
            if (is_pawn && (target >> 3) == (white ? 7 : 0))
                v += static_cast<unsigned>(promo < 0 ? QUEEN : promo + KNIGHT) << 6;
            if (mtype == KING || mtype == ROOK) v |= 1u << 9;
            put_word(w, source >> 3, v);
        }
        if ((rook & 7) == j && rook < 32)
            put_word(w, rook >> 3,
                     (pick_word(w, rook >> 3) & ~63u & 0xFFFu) + static_cast<unsigned>((white ? 0 : 56) + (dx > 0 ? 5 : 3)));
        // the en passant flag lives for one ply: clear every pawn's, set the double-stepper's
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if ((w[i] & 0x3C0u) == 0x200u) w[i] = w[i] & ~(1u << 9) & 0xFFFu;
        if (is_pawn && (dx == 16 || dx == -16) && (source & 7) == j)
            put_word(w, source >> 3, pick_word(w, source >> 3) | (1u << 9));
    }
    const unsigned rights_after = group_rights(w);
    const bool reset = captured < 32 || is_pawn;
    const int mag = reset ? 1 : (control < 0 ? -control : control) + 1;
    new_control = moves ? (white ? -mag : mag) : control;
    irreversible = moves && (reset || rights_after != rights_before);
}

// Key of a board.  The en passant file counts only when a capture is really available: a pawn of the
// mover stands beside the pawn that has just made its double step, and taking it does not leave the
// mover's king attacked.
__device__ __forceinline__ unsigned long long group_hash(const unsigned (&w)[4], const Board& b, bool black, int lane) {
    unsigned long long h = 0ull;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned word = w[i];
        const int type = (word >> 6) & 7, sq = word & 63;
        if ((word & 0x800u) == 0u) h ^= zobrist_key((((word & 0x400u) ? 6 : 0) + type) * 64 + sq);
    }
    // side to move and rights: one key each on lanes of their own
    const unsigned rights = group_rights(w);
    const int j = lane & 7;
    const bool own_key = j < 4 ? ((rights >> j) & 1u) != 0u : (j == 4 && black);
    if (own_key) h ^= zobrist_key(j < 4 ? ZOBRIST_CASTLE + j : ZOBRIST_SIDE);
    unsigned lo = static_cast<unsigned>(h), hi = static_cast<unsigned>(h >> 32);
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        lo ^= __shfl_xor_sync(kFull, lo, off);
        hi ^= __shfl_xor_sync(kFull, hi, off);
    }
    h = (static_cast<unsigned long long>(hi) << 32) | lo;
    if (b.ep_pawns != 0ull) {
        const unsigned long long victim = b.ep_pawns & (0ull - b.ep_pawns);
        const unsigned long long target = black ? victim >> 8 : victim << 8;
        bool legal = false;
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
            const unsigned long long capturer = side ? ((victim << 1) & ~kFileA) : ((victim >> 1) & ~kFileH);
            if ((capturer & b.my_pawns) != 0ull)
                legal |= !king_hit(b, black, ((b.occ & ~capturer) & ~victim) | target, victim);
        }
        if (legal) h ^= zobrist_key(ZOBRIST_EP + ((__ffsll(static_cast<long long>(victim)) - 1) & 7));
    }
    return h;
}

// kStep: play `move` first (or, with kPick, the floor(r * count)-th legal move of the incoming
// `mask` in (slot, square) order; a board without legal moves stays as it is) and write the new
// board, control word and irreversible flag; `mask` non-null: the legal words of the resulting
// board follow; `hash_out` non-null: its key.  In place (boards_out == boards) is safe: a board's
// lanes read all of it first.
template <bool kStep, bool kPick>
__global__ void __launch_bounds__(kEngineThreads) engine_group_kernel(
        const uint16_t* boards, const int16_t* control, const int* move,
        const signed char* promo, const float* r, int n, uint16_t* boards_out,
        int16_t* control_out, unsigned char* irreversible, unsigned long long* mask,
        unsigned char* in_check, int* move_out, unsigned long long* hash_out) {
    after_previous_grid();
    const int lane = threadIdx.x & 31, j = lane & 7;
    const long board = static_cast<long>(blockIdx.x) * kEngineBoards + (threadIdx.x >> 3);
    const bool valid = board < n;
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = valid ? boards[board * 32 + 8 * i + j] : 0x800u;
    int ctl = valid ? control[board] : 1;
    unsigned long long* words = mask + board * 32;
    const bool generate = mask != nullptr;
    bool moved = true;
    if (kStep) {
        int mv;
        if (kPick) {
            // this lane's legal words and, packed two counts to a register, their running totals
            // over the lanes: the order is slot-major, that is lane by lane within each i
            unsigned long long m[4];
            unsigned cnt[4], run[2];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                m[i] = valid ? words[8 * i + j] : 0ull;
                cnt[i] = __popcll(m[i]);
            }
            run[0] = cnt[0] | (cnt[1] << 16);
            run[1] = cnt[2] | (cnt[3] << 16);
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) {
                const unsigned a = __shfl_up_sync(kFull, run[0], off, 8), c = __shfl_up_sync(kFull, run[1], off, 8);
                if (j >= off) { run[0] += a; run[1] += c; }
            }
            const unsigned all0 = __shfl_sync(kFull, run[0], 7, 8), all1 = __shfl_sync(kFull, run[1], 7, 8);
            const int sum[4] = {static_cast<int>(all0 & 0xFFFFu), static_cast<int>(all0 >> 16),
                                static_cast<int>(all1 & 0xFFFFu), static_cast<int>(all1 >> 16)};
            const int total = sum[0] + sum[1] + sum[2] + sum[3];
            int pick = valid ? static_cast<int>(__fmul_rn(r[board], static_cast<float>(total))) : 0;
            pick = pick < total - 1 ? pick : total - 1;
            mv = 0x7fffffff;
            int before = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int upto = before + static_cast<int>((i & 1) ? run[i >> 1] >> 16 : run[i >> 1] & 0xFFFFu);
                int rest = pick - (upto - static_cast<int>(cnt[i]));
                if (total > 0 && rest >= 0 && pick < upto) {
                    unsigned long long v = m[i];
                    for (; rest > 0; --rest) v &= v - 1ull;
                    mv = (8 * i + j) * 64 + __ffsll(static_cast<long long>(v)) - 1;
                }
                before += sum[i];
            }
            mv = group_min(mv);
            if (mv == 0x7fffffff) mv = -1;
            moved = mv >= 0;
            if (move_out != nullptr && valid && j == 0) move_out[board] = mv;
        } else {
            mv = valid ? move[board] : -1;
        }
        int nc;
        bool irr;
        group_step(w, lane, ctl, mv, promo != nullptr && valid ? promo[board] : -1, nc, irr);
        if (valid && moved) {
            if (j == 0) {
                control_out[board] = static_cast<int16_t>(nc);
                if (irreversible != nullptr) irreversible[board] = irr ? 1 : 0;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) boards_out[board * 32 + 8 * i + j] = static_cast<uint16_t>(w[i]);
        }
        ctl = nc;
    }
    if (!generate && hash_out == nullptr) return;
    const bool black = ctl < 0;
    const Board b = board_planes(w, black);
    if (generate) {
        // a finished game of a playout keeps its (empty) legal words
        const bool chk = group_moves(w, b, black, lane, valid && moved, words);
        if (in_check != nullptr && valid && j == 0) in_check[board] = chk ? 1 : 0;
    }
    if (hash_out != nullptr) {
        const unsigned long long h = group_hash(w, b, black, lane);
        if (valid && j == 0) hash_out[board] = h;
    }
}

// How many of the first `length` entries of a game's ring equal `hash`: warp-collective.
constexpr int kMaxHistory = 100;
__device__ __forceinline__ int ring_matches(const unsigned long long* ring, long long length,
                                            unsigned long long hash, int lane) {
    const int len = static_cast<int>(length < kMaxHistory ? length : kMaxHistory);
    int c = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = 32 * k + lane;
        if (i < len) c += ring[i] == hash;
    }
    return static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(c)));
}

// Why a game is over (brokefish/env/torch_impl.py:632-676): 1 checkmate,
// 2 stalemate (no legal move, with or without check), else 3 when the control word's magnitude
// has reached 101 (fifty moves without capture or pawn move), else 4 when the position has
// occurred three times (`rep_count` when it is given, else counted in the game's `ring`; skipped
// without either), else 5 when neither side can mate -- no pawn, rook or queen and
// either no knight and every bishop on one colour of squares, or one knight and no bishop
// (torch_impl.py:604-629) -- else 0.  `result` is -1 for checkmate (the side to move lost), else 0.
//
// One WARP per game, lane = slot: a game's words, board and ring are contiguous runs that a warp
// reads whole, where a thread per game walked 1.1 KB of its own (4096 games with rings of up to
// forty entries: 4 us instead of 12 us for the two launches this one replaces).
__global__ void __launch_bounds__(128) terminal_kernel(const unsigned long long* mask,
                                                       const unsigned char* in_check,
                                                       const int16_t* control,
                                                       const uint16_t* boards,
                                                       const int* rep_count,
                                                       const unsigned long long* hash,
                                                       const unsigned long long* ring,
                                                       const long long* length, int n,
                                                       unsigned char* code, signed char* result) {
    after_previous_grid();
    const int lane = threadIdx.x & 31;
    const long board = static_cast<long>(blockIdx.x) * 4 + (threadIdx.x >> 5);
    if (board >= n) return;
    const unsigned word = boards[board * 32 + lane];
    const bool moves = __any_sync(kFull, mask[board * 32 + lane] != 0ull);
    int seen = rep_count != nullptr ? rep_count[board] : 1;
    if (ring != nullptr) seen += ring_matches(ring + board * kMaxHistory, length[board], hash[board], lane);
    const bool live = (word & 0x800u) == 0u;
    const int type = (word >> 6) & 7, sq = word & 63;
    const bool heavy = __any_sync(kFull, live && (type == PAWN || type == ROOK || type == QUEEN));
    const int knights = __popc(__ballot_sync(kFull, live && type == KNIGHT));
    const bool bishop = live && type == BISHOP;
    const int bishops = __popc(__ballot_sync(kFull, bishop));
    const int dark = __popc(__ballot_sync(kFull, bishop && (((sq & 7) + (sq >> 3)) & 1) == 0));
    if (lane != 0) return;
    const int c = control[board];
    int out = 0;
    if (!moves) out = in_check[board] ? 1 : 2;
    else if ((c < 0 ? -c : c) >= 101) out = 3;
    else if (seen >= 3) out = 4;
    else if (!heavy && ((knights == 0 && (dark == 0 || dark == bishops)) || (knights == 1 && bishops == 0))) out = 5;
    code[board] = static_cast<unsigned char>(out);
    if (result != nullptr) result[board] = out == 1 ? -1 : 0;
}

// The per-game repetition ring (brokefish/env/torch_impl.py:571-602): `ring` [n,100] position keys
// since the last irreversible move, `length` [n].  Push: record the position being left (`hash`
// is the key BEFORE the move, `irreversible` describes the move); an irreversible move empties
// the ring, because nothing at or before it can recur.
__global__ void __launch_bounds__(128) history_push_kernel(unsigned long long* ring,
                                                           long long* length,
                                                           const unsigned long long* hash,
                                                           const unsigned char* irreversible, int n) {
    after_previous_grid();
    const long g = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (g >= n) return;
    if (irreversible[g]) { length[g] = 0; return; }
    const long long len = length[g];
    ring[g * kMaxHistory + (len < kMaxHistory - 1 ? len : kMaxHistory - 1)] = hash[g];
    length[g] = len + 1 < kMaxHistory ? len + 1 : kMaxHistory;
}
// The same into new arrays: one pass copies the ring and puts the key in its place.  Bound by memory
// (1,632 bytes per game); a thread copies 16 bytes (a ring is fifty of them), or 8 where an array
// does not start on a 16-byte boundary.
template <int kWords>
__global__ void __launch_bounds__(256) history_push_to_kernel(const unsigned long long* ring,
                                                              const long long* length,
                                                              const unsigned long long* hash,
                                                              const unsigned char* irreversible, int n,
                                                              unsigned long long* new_ring,
                                                              long long* new_length) {
    after_previous_grid();
    constexpr unsigned kPieces = kMaxHistory / kWords;
    const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long g = i / kPieces;
    const int piece = static_cast<int>(i - g * kPieces);
    if (g >= n) return;
    unsigned long long v[kWords];
    if constexpr (kWords == 2) {
        const ulonglong2 t = reinterpret_cast<const ulonglong2*>(ring)[i];
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = ring[i];
    }
    const bool empties = irreversible[g] != 0;
    const long long len = length[g];
    const int at = empties ? -1 : static_cast<int>(len < kMaxHistory - 1 ? len : kMaxHistory - 1);
#pragma unroll
    for (int k = 0; k < kWords; ++k)
        if (piece * kWords + k == at) v[k] = hash[g];
    if constexpr (kWords == 2) reinterpret_cast<ulonglong2*>(new_ring)[i] = make_ulonglong2(v[0], v[1]);
    else new_ring[i] = v[0];
    if (piece == 0) new_length[g] = empties ? 0 : (len + 1 < kMaxHistory ? len + 1 : kMaxHistory);
}
// How many times the position has occurred, counting the present one: one warp per game.
__global__ void __launch_bounds__(128) repetition_kernel(const unsigned long long* hash,
                                                         const unsigned long long* ring,
                                                         const long long* length, int n,
                                                         int* count) {
    after_previous_grid();
    const int lane = threadIdx.x & 31;
    const long g = static_cast<long>(blockIdx.x) * 4 + (threadIdx.x >> 5);
    if (g >= n) return;
    const int c = 1 + ring_matches(ring + g * kMaxHistory, length[g], hash[g], lane);
    if (lane == 0) count[g] = c;
}

}  // namespace bfmg
