// The evaluator kernel on tensor-core tiles of one or two boards, by pairs of SMs (included by bf_encoder.cu): the
// form every plain evaluation runs in.
//
// Why one or two boards, and why pairs.  A 128-row tile takes as long as one board's chain of phases, with four warps
// to a board; sixteen row warps on one or two boards make that chain a quarter as long.  A product then
// has 32 or 64 rows, and two things bound it: the weights' way out of shared memory (an N = 256 product of 64 rows
// by `tcgen05.mma.ws` takes 80.7 cycles per 32 bytes of K, of which the weights are 64) and their way into the SM (at
// 64 bytes a cycle, 12.3 k cycles of a layer in int8, 24.6 k in fp16).  `tcgen05.mma.cta_group::2` halves
// both: two SMs share a product, M = 128 rows, 64 of each; each loads and keeps half of the weight rows (64.8 cycles per
// 32 bytes of K).  An SM's tensor memory gets the product of its own rows over all 128 lanes: lane quadrant q holds
// rows 32 (q & 1) .. + 31 and output columns 128 (q >> 1) .. + 127.  So sixteen row warps (four per quadrant,
// thread = row x 32 columns) share the element-wise work of two boards; a single board's operand rows are there
// twice, and the two quadrants that hold its product take half of the columns each (thread = row x 16).
//
// What follows from a thread's columns being the same in every product:
//   * the residual stream x stays in the owning thread's registers from the embedding to the heads;
//   * all of tensor memory is accumulators: four slots of one N = 256 product.  Q, K, V, out-projection
//     take slots 0-3, the four hidden chunks of ff1 slots 0-3, their ff2 products the slot of the
//     chunk they come from, so every product of a phase is issued as soon as its operand is there
//     and no slot needs an "empty" barrier: the operand that starts a product is published by warps
//     that have read what was in its slot;
//   * with two boards a thread holds a whole head's row (32 columns) of Q, K and V: attention needs
//     no other warp, only a 2 KB scratch block per warp.
//
// The arithmetic is the four-board kernel's, bit for bit (the order of every sum included).
//
// Measured on one B200, us, against tiles of one SM (M = 32 and 64 by `tcgen05.mma.ws`): a one-board tile
// int8 86 (91), e4m3 94 (101), fp16 105 to 110 (129); a two-board tile 116 (127), 117 (130), 121 to 126 (152); batch 4096 1560
// (1677), 1576 (1735), 1764 (1877, then on four-board tiles; 1620 before the power cap).  What bounds it: the row warps, four to
// a scheduler and all in the same phase, at 61 % of the issue slots in int8; of a one-board tile's 19,300 cycles per layer a
// row warp waits 4,400 for products, of a two-board tile's 26,500 5,700.  In fp16 and e4m3 a loop of large batches also runs
// into the 1000 W power cap (1.75 to 1.87 GHz; int8 stays at 890 W and 1.965 GHz).
#pragma once

namespace bf {
namespace ws {

constexpr int kProducerWarp = 16, kMmaWarp = 17, kExpandWarp = 18;
// (two-board tiles: a whole warpgroup of the warps that give registers up)
constexpr int threads(bool expand, int boards) { return expand || boards == 2 ? 640 : 576; }
// Two-board tiles: a row warp's registers and another's, out of the 96 a thread that the launch comes with.  4096
// positions int8 1570 us without the split, 1543 with it; 112 and 32 are too few for the producer (e4m3 +2 %, fp16 +10 %),
// and one-board tiles, which need 95, lose 1 % by it.
constexpr int kRowRegisters = 104, kHelperRegisters = 64, kLaunchRegisters = 96;
static_assert(16 * kRowRegisters + 4 * kHelperRegisters <= 20 * kLaunchRegisters, "a larger share would be waited for in vain");
constexpr uint32_t kStage = 16384;                 // one 128-byte K-slab of this SM's 128 rows of a product's weights
// ---- shared memory map ------------------------------------------------------------------
// A operand: K-slabs of [rows][128 B], two of bytes or (where QKV or the out-projection runs in fp16)
// four of halves.  H: the ff2 operand's chunks; before and after that the attention scratch, the norms'
// partial sums, the head operand.
template <int kAr>
struct Map {
    static constexpr int kStages = Cfg<kAr>::kHalfA ? 6 : 8;
    static constexpr uint32_t SM_H = Cfg<kAr>::kHalfA ? 32768 : 16384;
    static constexpr uint32_t SM_RING = SM_H + 65536;
};
constexpr uint32_t SM_A = 0;
constexpr uint32_t kHeadA = 32768;                 // the head operand's place in H, clear of the other board's partial sums
// the fused expansion's logits: per board 32 policy rows of 128 bytes, then 16 bytes of promotion logits
// per slot; the last quarter of H, which the next tile touches in its first FFN
constexpr uint32_t kStagePolicy = 49152, kStageAux = kStagePolicy + 8192;
constexpr uint32_t SM_STAT = 16384 + 65536 + 8 * kStage;
constexpr uint32_t SM_MAX = SM_STAT + 1024;        // row maxima: attention output, four hidden chunks
constexpr uint32_t SM_LIST = SM_MAX + 5 * 256;     // fused expansion: a list per board
constexpr uint32_t SM_PAR = SM_LIST + 2 * kListBytes;        // scales and biases of two layers
constexpr uint32_t SM_BAR = SM_PAR + 2 * kLparamStride;
constexpr uint32_t SM_MISC = SM_BAR + 8 * 34;
constexpr uint32_t SM_BYTES = SM_MISC + 64, kSmemRequest = SM_BYTES + 1024;
static_assert(kSmemRequest <= 232448 && kLparamStride % 16 == 0 && SM_PAR % 16 == 0, "shared memory map");
static_assert(Map<kArF16>::SM_RING + 6 * kStage <= SM_STAT && Map<kArInt8>::SM_RING + 8 * kStage <= SM_STAT, "shared memory map");
enum { B_FULL = 0, B_EMPTY = 8, B_ACC = 16, B_PAR = 20, B_A = 22, B_H = 23, B_MAX = 27, B_STAGED = 31, B_EXPANDED = 32, B_COUNT = 33 };
__device__ __forceinline__ uint32_t bar(uint32_t smem, int i) { return smem + SM_BAR + 8u * i; }

// ---- what is different in a pair of SMs ----
// A product is the pair's (`umma_pair_*`), its completion goes to the same barrier in both SMs (`tc_commit_pair`), and an
// operand's or a weight stage's arrival to the first SM's barrier, whose MMA warp issues the pair's products.  What crosses
// from SM to SM -- an operand's rows, a weight stage -- is written or copied into the writer's own shared memory and read by the
// product's asynchronous proxy: a writer's proxy fence, the arrival's release and the MMA warp's acquire at cluster scope.
__device__ __forceinline__ void mbar_arrive_first(uint32_t bar) { mbar_arrive_cluster(cluster_address(bar, 0)); }

// Which boards a CTA evaluates, tile by tile.  A launch's tiles hold `NB` boards each.  At most `one_most` boards
// per CTA: one-board tiles alone.  More: as many whole waves of two-board tiles as there are, then what is left, one board
// per CTA where that is enough (and allowed), else two.  A one-board tile takes about two thirds of a
// two-board tile's time.  The two forms are kernels of their own -- together they cost each other registers, 2 to
// 4 % of a tile -- so that a batch takes one launch of either or one of each; of a leaf list, whose length only the
// kernels know, each makes its own part.  `grid`: CTAs of a whole wave.  Both SMs of a pair have as many tiles.
template <int NB>
struct Tiles {
    int n, first, step, tiles;       // boards in all; this CTA's first board; boards per round; rounds
    __device__ Tiles(int n_, int grid, int ctas, int cta, int one_most) : n(n_) {
        const int full = n / (2 * grid), rest = n - full * 2 * grid, lead = cta & ~1;
        const bool singles = n <= one_most * grid, one = rest <= grid && one_most > 0;
        int begin = 0, end = n;      // the boards of this form
        if (NB == 1) { if (!singles) begin = one ? n - rest : n; }
        else if (singles) end = 0;
        else if (one) end = n - rest;
        step = NB * ctas;
        first = begin + NB * cta;
        const int mine = begin + NB * lead;
        tiles = mine < end ? (end - mine + step - 1) / step : 0;
    }
    __device__ int count() const { return tiles; }
    __device__ int at(int k) const { return first + k * step; }
};

struct Row {
    int lane, q, s;             // lane quadrant, warp within the quadrant
    uint32_t smem, tm;          // tm: tensor memory with this warp's lane offset
    uint8_t* smem_gen;
    volatile int* abort_flag;
    uint64_t one2;
    uint32_t layers, tiles;     // layers and tiles finished so far: a slot's barrier completes `completions`
                                // times per layer, and slot 0's once per tile for the heads
    int n;
    uint32_t h;                 // shared address of H
    __device__ uint32_t a() const { return smem + SM_A; }
};

// A tile of NB boards as its thread sees it.
template <int NB>
struct Own {
    static constexpr int kW = 16 * NB;                       // columns per thread of a 256-wide row
    static constexpr uint32_t kSlab = 64 * 128;              // bytes of a K-slab of an operand
    static constexpr uint32_t kSlot = 128;                   // tensor-memory columns of a slot
    static constexpr int kGroup = 16 / NB;                   // threads that share a row
    static __device__ int board(const Row& c) { return NB == 1 ? 0 : c.q & 1; }
    static __device__ int col(const Row& c) { return 128 * (c.q >> 1) + 32 * c.s + (NB == 1 ? 16 * (c.q & 1) : 0); }
    static __device__ int member(const Row& c) { return NB == 1 ? 8 * (c.q >> 1) + 2 * c.s + (c.q & 1) : 4 * (c.q >> 1) + c.s; }
    static __device__ int row(const Row& c) { return 32 * board(c) + c.lane; }
    static __device__ uint32_t slot(const Row& c, int k) { return c.tm + kSlot * k + 32 * c.s + (NB == 1 ? 16 * (c.q & 1) : 0); }
};
// 16 bytes of an operand row.  A single board's rows are there twice, so that every quadrant of tensor memory has them.
template <int NB>
__device__ __forceinline__ void store_operand(uint32_t at, uint4 v) {
    sts128(at, v);
    if (NB == 1) sts128(at + 32 * 128, v);
}
// The warps of a board meet here (barriers of their own for one- and two-board tiles: a warp may be a
// tile ahead).
template <int NB>
__device__ __forceinline__ void board_sync(const Row& c) { __syncwarp(); named_bar_sync(NB == 1 ? 11 : 1 + Own<NB>::board(c), 512 / NB); }

// The two warps of a head (one-board tiles).
__device__ __forceinline__ void pair_sync(int head) { __syncwarp(); named_bar_sync(3 + head, 64); }

// How often a slot's barrier completes in a layer: with Q, K, V or the out-projection, with ff1's chunk,
// with ff2's (in fp16, whose ff2 has one sum, slots 0 and 1 with its first and second chunk and slot 2 with all of
// it).  Every completion is one that all row warps wait for: a parity wait tells a phase only from the one before it.
template <int kAr>
__host__ __device__ constexpr uint32_t completions(int slot) { return kAr == kArF16 && slot == 3 ? 2u : 3u; }
// The `use`-th of them in this layer; of slot 0, use 0 after the last layer is the heads' product.
template <int kAr>
__device__ __forceinline__ void wait_acc(const Row& c, int slot, int use) {
    const uint32_t n = completions<kAr>(slot) * c.layers + use + (slot == 0 ? c.tiles : 0u);
    mbar_wait(bar(c.smem, B_ACC + slot), n & 1u, c.abort_flag, kErrRowAcc);
    __syncwarp();                                            // what follows is for a converged warp
    tc_fence_after();
}
// The scales and biases of the layer this thread is at (two copies, filled by the weight stream a layer
// ahead): shared address of the layer's block.  Read through L1, beside 228 KB of shared memory, they
// cost 3 to 6 % of a tile more.
__device__ __forceinline__ uint32_t layer_params(const Row& c) {
    return c.smem + SM_PAR + (c.layers & 1u) * kLparamStride;
}
__device__ __forceinline__ void wait_params(const Row& c) {
    mbar_wait(bar(c.smem, B_PAR + (c.layers & 1u)), (c.layers >> 1) & 1u, c.abort_flag, kErrRowAcc);
    __syncwarp();
}
// This warp's operand rows are written and what it read of tensor memory has arrived: publish.
__device__ __forceinline__ void publish(const Row& c, int b) {
    tc_fence_before();
    fence_proxy_async_smem();
    __syncwarp();
    if (c.lane == 0) mbar_arrive_first(bar(c.smem, b));
}
__device__ __forceinline__ float lds_f(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds_u(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t lds_u64(uint32_t addr) {
    uint64_t v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}
// Row maxima of non-negative values meet in shared memory by an integer maximum of their bits.
__device__ __forceinline__ void max_to(uint32_t addr, float v) {
    asm volatile("red.shared.max.u32 [%0], %1;" ::"r"(addr), "r"(__float_as_uint(v)) : "memory");
}
// The same for a hidden chunk, whose maxima are waited for later: the warp has given its part.
__device__ __forceinline__ void max_to(uint32_t addr, float v, const Row& c, int chunk) {
    max_to(addr, v);
    __syncwarp();
    if (c.lane == 0) mbar_arrive(bar(c.smem, B_MAX + chunk));
}
// The chunk's maxima are all there.
template <int NB>
__device__ __forceinline__ void board_sync(const Row& c, int chunk) {
    mbar_wait(bar(c.smem, B_MAX + chunk), c.layers & 1u, c.abort_flag, kErrRowAcc);
    __syncwarp();
}
// A row's scale amax / Q and its reciprocal, both correctly rounded, amax being a non-negative fp16 value.  The
// scale is a product with 1 / Q held in two words (Brisebarre and Muller 2008), the upper one rounded down so
// that an infinite amax, a row that has overflowed, stays infinite; the reciprocal one Newton step on the
// hardware's, the residual taken by fma (Markstein 1990), its minimum leaving infinity's reciprocal zero.
// Every fp16 amax gives the bits of `__fdiv_rn` for each of the three ranges, as does the reciprocal of
// every fp32 value from 1 to 32, a softmax row's sum (`scales_kernel`).  Two divisions one after the other
// took 300 cycles, this takes 45.
struct Scale { float scale, inverse; };
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float reciprocal(float x) {
    const float y = rcp_approx(x);
    return __fmaf_rn(__fmaf_rn(-x, y, 1.0f), y, y);
}
__device__ __forceinline__ Scale with_inverse(float sc) {
    const float y = rcp_approx(sc);
    return {sc, __fmaf_rn(fminf(__fmaf_rn(-sc, y, 1.0f), 1.0f), y, y)};
}
__device__ __forceinline__ Scale scale_s8(float amax) {
    constexpr float hi = 0x1.020408p-7f, lo = static_cast<float>(1.0 / kQMaxS8 - hi);
    return with_inverse(amax > 0.f ? __fmaf_rn(amax, hi, __fmul_rn(amax, lo)) : 1.0f);
}
__device__ __forceinline__ Scale scale_u8(float amax) {
    constexpr float hi = 0x1.01010p-8f, lo = static_cast<float>(1.0 / kQMaxU8 - hi);
    return with_inverse(amax > 0.f ? __fmaf_rn(amax, hi, __fmul_rn(amax, lo)) : 1.0f);
}
__device__ __forceinline__ Scale scale_e4m3(float amax) {
    return with_inverse(amax > 0.f ? __fmul_rn(amax, 1.0f / kQMaxE4M3) : 1.0f);      // a power of two: exact
}
// Sixteen columns' biases (a broadcast: a warp's threads share their columns).
struct Bias { uint4 lo, hi; };
__device__ __forceinline__ Bias load_bias(uint32_t addr) { return {lds128(addr), lds128(addr + 16)}; }
// `(float(acc) * sa) * sw` -> fp16, + fp16 bias, optional ReLU, for sixteen columns: `descale`'s arithmetic.
template <bool kRelu, int kAcc>
__device__ __forceinline__ void descale16(const uint32_t (&acc)[16], float sa, float sw, const Bias& bias, uint32_t* out) {
    const uint32_t bw[8] = {bias.lo.x, bias.lo.y, bias.lo.z, bias.lo.w, bias.hi.x, bias.hi.y, bias.hi.z, bias.hi.w};
    const uint64_t sw2 = pk2(sw, sw);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint32_t h;
        if (kAcc == kAccPlain) {
            h = __byte_perm(acc[2 * i], acc[2 * i + 1], 0x5410);
        } else {
            const float a0 = kAcc == kAccInt ? static_cast<float>(static_cast<int>(acc[2 * i])) : __uint_as_float(acc[2 * i]);
            const float a1 = kAcc == kAccInt ? static_cast<float>(static_cast<int>(acc[2 * i + 1])) : __uint_as_float(acc[2 * i + 1]);
            h = f2_to_h2(mul2(pk2(__fmul_rn(a0, sa), __fmul_rn(a1, sa)), sw2));
        }
        out[i] = kRelu ? hfma2_relu(h, 0x3C003C00u, bw[i]) : as_u32(__hadd2(as_h2(h), as_h2(bw[i])));
    }
}
// This thread's columns of a slot, 16 at a time: `use(piece, words)`.  No load is left in flight while
// another piece is worked on: the registers that one lands in are then free of pressure from the code
// around them, and the scheduler's other warps cover its latency.
template <int NB, class F>
__device__ __forceinline__ void each_piece(uint32_t t, F&& use) {
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        uint32_t acc[16];
        tmem_ld16(t + 16 * k, acc);
        tmem_wait_ld();
        use(k, acc);
    }
}
// Piece k (16 columns) of this thread's columns into an operand: quantised to bytes (two K-slabs), or as
// fp16 (four).
template <int NB, bool kE4M3 = false>
__device__ __forceinline__ void store_operand8(const Row& c, uint32_t base, int k, const uint32_t* v, float inv) {
    using O = Own<NB>;
    const int col = O::col(c);
    store_operand<NB>(base + (col >> 7) * O::kSlab + sw_off(O::row(c), ((col & 127) >> 4) + k), quant16_any<kE4M3>(v, inv, c.one2));
}
template <int NB>
__device__ __forceinline__ void store_operand16(const Row& c, uint32_t base, int k, const uint32_t* v) {
    using O = Own<NB>;
    const int col = O::col(c), row = O::row(c), group = ((col & 63) >> 3) + 2 * k;
    const uint32_t slab = base + (col >> 6) * O::kSlab;
    store_operand<NB>(slab + sw_off(row, group), make_uint4(v[0], v[1], v[2], v[3]));
    store_operand<NB>(slab + sw_off(row, group + 1), make_uint4(v[4], v[5], v[6], v[7]));
}

// ---- LayerNorm ----
// Partial sums of eight columns each, then the butterfly 16, 8, 4, 2, 1 over the row's 32 partials,
// in the reference's order (see `ln_stage`).  A row's partials meet in shared memory; a few of the
// board's warps, eight rows each, then finish them -- four lanes to a row: sums and squares, each
// with half of what the member threads' order leaves after the butterfly's outer levels, which are plain
// additions in the lane -- and leave mean, 1/sqrt, 1/scale and scale for everybody.  (Every thread reading
// all of its row's partials instead is 1,500 cycles of shared-memory bandwidth per norm; all sixteen
// warps finishing two to four rows each put the same chain of 90 instructions into every scheduler
// four times over, 780 cycles.)
template <int NB, int kAr>
__device__ __forceinline__ float4 row_statistics(const Row& c, const Params& p, const uint32_t (&x)[8 * NB]) {
    using O = Own<NB>;
    constexpr uint32_t kSquares = 8 * 512 + 64;                 // NB == 2: the squares' offset (other banks)
    constexpr uint32_t kMinMax = 12288;
    const uint32_t base = c.h + 16384u * O::board(c);
    const int t = O::member(c);
    {
        uint64_t s2[NB], q2[NB];
#pragma unroll
        for (int pr = 0; pr < NB; ++pr) {
            float sa = 0.f, sb = 0.f, qa = 0.f, qb = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                sum_h2(x[8 * pr + k], sa, qa);
                sum_h2(x[8 * pr + 4 + k], sb, qb);
            }
            s2[pr] = pk2(sa, sb);
            q2[pr] = pk2(qa, qb);
        }
        __half2 mn = as_h2(x[0]), mx = as_h2(x[0]);
#pragma unroll
        for (int i = 1; i < 8 * NB; ++i) {
            mn = __hmin2(mn, as_h2(x[i]));
            mx = __hmax2(mx, as_h2(x[i]));
        }
        const uint32_t at = base + 512u * t + 16u * c.lane;
        float a0, a1, b0, b1;
        upk2(s2[0], a0, a1);
        if constexpr (NB == 1) {
            upk2(q2[0], b0, b1);
            sts_f4(at, make_float4(a0, a1, b0, b1));
        } else {
            upk2(s2[1], b0, b1);
            sts_f4(at, make_float4(a0, a1, b0, b1));
            upk2(q2[0], a0, a1);
            upk2(q2[1], b0, b1);
            sts_f4(at + kSquares, make_float4(a0, a1, b0, b1));
        }
        // (minimum, -maximum): one packed minimum reduces both
        const __half2 lo = __lows2half2(mn, __hneg2(mx)), hi = __highs2half2(mn, __hneg2(mx));
        sts32(base + kMinMax + 128u * t + 4u * c.lane, as_u32(__hmin2(lo, hi)));
    }
    board_sync<NB>(c);
    if (c.s < NB) {
        const int lane = c.lane, j = lane & 3;                           // j: bit 1 squares, bit 0 which half
        const int r = 8 * (NB == 1 ? c.q : 2 * (c.q >> 1) + c.s) + (lane >> 2);
        float v;
        if constexpr (NB == 1) {
            // levels 16 and 8 over the quadrants, 4 and 2 over s, 1 over the thread's two partials
            const uint32_t at = base + 16u * r + 4u * j;
            float m[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                m[k] = __fadd_rn(__fadd_rn(lds_f(at + 512u * k), lds_f(at + 512u * (k + 8))),
                                 __fadd_rn(lds_f(at + 512u * (k + 4)), lds_f(at + 512u * (k + 12))));
            v = __fadd_rn(__fadd_rn(m[0], m[2]), __fadd_rn(m[1], m[3]));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
        } else {
            // levels 16, 8 and 4 over the members, 2 over the halves of their four partials, 1 in the lane
            const uint32_t at = base + (j >> 1) * kSquares + 16u * r + 8u * (j & 1);
            uint64_t m[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) m[k] = lds_u64(at + 512u * k);
#pragma unroll
            for (int k = 0; k < 4; ++k) m[k] = add2(m[k], m[k + 4]);
            float a, b;
            upk2(add2(add2(m[0], m[2]), add2(m[1], m[3])), a, b);
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 1));
            b = __fadd_rn(b, __shfl_xor_sync(0xffffffffu, b, 1));
            v = __fadd_rn(a, b);
        }
        __half2 mm = as_h2(lds_u(base + kMinMax + 128u * j + 4u * r));
#pragma unroll
        for (int k = 4; k < O::kGroup; k += 4) mm = __hmin2(mm, as_h2(lds_u(base + kMinMax + 128u * (j + k) + 4u * r)));
        mm = __hmin2(mm, as_h2(__shfl_xor_sync(0xffffffffu, as_u32(mm), 1)));
        mm = __hmin2(mm, as_h2(__shfl_xor_sync(0xffffffffu, as_u32(mm), 2)));
        const float other = __shfl_xor_sync(0xffffffffu, v, 2);
        const float tot = (j & 2) ? other : v, totq = (j & 2) ? v : other;
        const float xmin = __low2float(mm), xmax = -__high2float(mm);
        const float mean = __fmul_rn(tot, 1.0f / 256.0f);
        const float var = fmaxf(__fsub_rn(__fmul_rn(totq, 1.0f / 256.0f), __fmul_rn(mean, mean)), 0.f);
        const float rstd = p.rsqrt_rn ? __frsqrt_rn(__fadd_rn(var, p.eps)) : rsqrtf(__fadd_rn(var, p.eps));
        const float e_lo = __half2float(__float2half_rn(__fmul_rn(__fsub_rn(xmin, mean), rstd)));
        const float e_hi = __half2float(__float2half_rn(__fmul_rn(__fsub_rn(xmax, mean), rstd)));
        const float amax = fmaxf(fabsf(e_lo), fabsf(e_hi));
        const Scale sc = kAr == kArE4M3 ? scale_e4m3(amax) : scale_s8(amax);
        if (j == 0) sts_f4(c.smem + SM_STAT + 16u * (32 * O::board(c) + r), make_float4(-mean, rstd, sc.inverse, sc.scale));
    }
    board_sync<NB>(c);
    return lds_f4(c.smem + SM_STAT + 16u * O::row(c));
}

// An attention or FFN norm: x_hat = fp16((x - mean) * rstd) into the A operand, quantised (returns the
// row's scale) or as it is.
template <int NB, int kAr>
__device__ __forceinline__ float norm_to_operand(const Row& c, const Params& p, const uint32_t (&x)[8 * NB], bool as_f16) {
    const float4 st = row_statistics<NB, kAr>(c, p, x);
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float a, b;                     // (scalar multiplies: half a per cent faster than a packed one)
            upk2(add_h2_f(x[8 * k + i], st.x), a, b);
            v[i] = pack_h2(__fmul_rn(a, st.y), __fmul_rn(b, st.y));
        }
        if (kAr != kArInt8 && kAr != kArI8Qkv && as_f16) store_operand16<NB>(c, c.a(), k, v);
        else store_operand8<NB, kAr == kArE4M3>(c, c.a(), k, v, st.z);
    }
    publish(c, B_A);
    return st.w;
}

// ---- attention ----
// A head's 32 rows of 32 halves in a 2 KB block: 64-byte rows, 16-byte groups moved by the row pair so
// that eight rows of one group (what ldmatrix and a warp's stores touch at a time) hit all banks.
__device__ __forceinline__ uint32_t head_off(int row, int group) {
    return static_cast<uint32_t>(row) * 64u + (static_cast<uint32_t>(group ^ ((row >> 1) & 3)) << 4);
}
// Scores of 16 query rows (fragments qa) against the head's 32 keys, softmax, probabilities as A
// fragments: `attention_unit`'s arithmetic.
__device__ __forceinline__ void scores(const uint32_t (&qa)[2][4], uint32_t ks, int lane, uint32_t (&s)[4][2]) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        s[nt][0] = s[nt][1] = 0u;
        uint32_t kb[4];
        ldmatrix_x4(kb, ks + head_off(8 * nt + (lane & 7), lane >> 3));
        mma_f16_f16(s[nt], qa[0], kb[0], kb[1]);      // dims 0-15, then 16-31
        mma_f16_f16(s[nt], qa[1], kb[2], kb[3]);
    }
}
__device__ __forceinline__ void softmax(uint32_t (&s)[4][2], const uint32_t (&dead)[4]) {
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
        float pv[4][2];
        __half2 val[4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) val[nt] = __hadd2(as_h2(s[nt][hi]), as_h2(dead[nt]));
        const __half2 m2 = __hmax2(__hmax2(val[0], val[1]), __hmax2(val[2], val[3]));
        float mx = fmaxf(__low2float(m2), __high2float(m2));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        float sum = 0.f;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            upk2(add_h2_f(as_u32(val[nt]), -mx), pv[nt][0], pv[nt][1]);
            pv[nt][0] = __expf(pv[nt][0]);           // an all-dead row keeps the reference's NaN
            pv[nt][1] = __expf(pv[nt][1]);
            sum += pv[nt][0] + pv[nt][1];
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        const float inv = reciprocal(sum);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) s[nt][hi] = pack_h2(pv[nt][0] * inv, pv[nt][1] * inv);
    }
}
__device__ __forceinline__ void load_query(uint32_t (&qa)[2][4], uint32_t qs, int first, int lane) {
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) ldmatrix_x4(qa[kk], qs + head_off(first + (lane & 15), 2 * kk + (lane >> 4)));
}
__device__ __forceinline__ void weighted_values(const uint32_t (&s)[4][2], uint32_t vs, int lane, uint32_t (&o)[4][2]) {
    uint32_t pa[2][4];
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
        pa[kk][0] = s[2 * kk][0];     pa[kk][1] = s[2 * kk][1];
        pa[kk][2] = s[2 * kk + 1][0]; pa[kk][3] = s[2 * kk + 1][1];
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        o[nt][0] = o[nt][1] = 0u;
        uint32_t vb[4];
        ldmatrix_x4_trans(vb, vs + head_off(lane, nt));
        mma_f16_f16(o[nt], pa[0], vb[0], vb[1]);      // keys 0-15, then 16-31
        mma_f16_f16(o[nt], pa[1], vb[2], vb[3]);
    }
}
__device__ __forceinline__ void store_outputs(const uint32_t (&o)[4][2], uint32_t os, int first, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        sts32(os + head_off(first + g, nt) + 4 * t, o[nt][0]);
        sts32(os + head_off(first + g + 8, nt) + 4 * t, o[nt][1]);
    }
}

// This thread's columns of product `m` (0 Q, 1 K, 2 V) as fp16 into its head's block.
template <int NB, int kAr>
__device__ __forceinline__ void stage_qkv(const Row& c, uint32_t lp, float sa, int m, uint32_t block) {
    using O = Own<NB>;
    const int col = O::col(c);
    const uint32_t bias_at = lp + LP_B_QKV + 2u * ((col >> 6) * 192 + m * 64 + (col & 63));
    const float sw = lds_f(lp + LP_SW_QKV + 4u * (m * 2 + (col >> 7)));
    Bias bias = load_bias(bias_at);
    wait_acc<kAr>(c, m, 0);
    each_piece<NB>(O::slot(c, m), [&](int k, const uint32_t (&acc)[16]) {
        uint32_t h[8];
        if (k > 0) bias = load_bias(bias_at + 32 * k);
        descale16<false, Cfg<kAr>::kQkvF16 ? kAccPlain : kAccInt>(acc, sa, sw, bias, h);
        if (k == 0) __syncwarp();
        const int group = ((col & 31) >> 3) + 2 * k;
        sts128(block + head_off(c.lane, group), make_uint4(h[0], h[1], h[2], h[3]));
        sts128(block + head_off(c.lane, group + 1), make_uint4(h[4], h[5], h[6], h[7]));
    });
}

template <int NB, int kAr>
__device__ __forceinline__ void attention_block(const Row& c, uint32_t lp, float sa, uint32_t alive, uint32_t (&x)[8 * NB]) {
    using O = Own<NB>;
    const int lane = c.lane, col = O::col(c);
    uint32_t dead[4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        const uint32_t two = (alive >> (8 * nt + 2 * (lane & 3))) & 3u;
        dead[nt] = ((two & 1u) ? 0u : 0xfc00u) | ((two & 2u) ? 0u : 0xfc000000u);
    }
    uint32_t oh[8 * NB];
    // Q, K and V one after the other.  Two boards: one warp per head, whose block serves Q, K, V and the
    // outputs in turn.  One board: two warps per head, each with half the query rows; Q, K and V have
    // blocks of their own and the outputs go over Q.
    const int head = NB == 1 ? 4 * (c.q >> 1) + c.s : 4 * c.q + c.s;
    const int first = NB == 1 ? 16 * (c.q & 1) : 0;
    const uint32_t block = c.h + 2048u * head;
    uint32_t qa[NB][2][4], s[NB][4][2];
#pragma unroll
    for (int u = 0; u < NB; ++u) {
#pragma unroll
        for (int i = 0; i < 8; ++i) { qa[u][i >> 2][i & 3] = 0u; s[u][i >> 1][i & 1] = 0u; }
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const uint32_t at = NB == 1 ? block + 16384u * m : block;
        stage_qkv<NB, kAr>(c, lp, sa, m, at);
        if (NB == 1) { if (m > 0) pair_sync(head); } else __syncwarp();
        if (m == 0) {
            if (NB == 2) {
                load_query(qa[0], at, 0, lane);
                load_query(qa[NB - 1], at, 16, lane);
            }
        } else if (m == 1) {
            if (NB == 1) load_query(qa[0], block, first, lane);
#pragma unroll
            for (int u = 0; u < NB; ++u) scores(qa[u], at, lane, s[u]);
#pragma unroll
            for (int u = 0; u < NB; ++u) softmax(s[u], dead);
        } else {
            uint32_t o[NB][4][2];
#pragma unroll
            for (int u = 0; u < NB; ++u) weighted_values(s[u], at, lane, o[u]);
            __syncwarp();
#pragma unroll
            for (int u = 0; u < NB; ++u) store_outputs(o[u], block, first + 16 * u, lane);
        }
    }
    if (NB == 1) pair_sync(head); else __syncwarp();
#pragma unroll
    for (int k = 0; k < 2 * NB; ++k) {
        const uint4 v = lds128(block + head_off(lane, ((col & 31) >> 3) + k));
        oh[4 * k] = v.x; oh[4 * k + 1] = v.y; oh[4 * k + 2] = v.z; oh[4 * k + 3] = v.w;
    }
    // the attention output is the out-projection's operand: quantised by its row maximum, or as it is
    Scale so = {1.f, 1.f};
    if constexpr (Cfg<kAr>::kOutF16) {
#pragma unroll
        for (int k = 0; k < NB; ++k) store_operand16<NB>(c, c.a(), k, &oh[8 * k]);
    } else {
        const uint32_t m = c.smem + SM_MAX + 4u * O::row(c);
        max_to(m, amax_h2<8 * NB>(oh, true));
        board_sync<NB>(c);
        so = scale_s8(lds_f(m));
#pragma unroll
        for (int k = 0; k < NB; ++k) store_operand8<NB>(c, c.a(), k, &oh[8 * k], so.inverse);
    }
    publish(c, B_A);
    // x = fp16(x + fp16(fp16(descale) + b_o))
    const float sw = lds_f(lp + LP_SW_O + 4u * (col >> 7));
    Bias bias = load_bias(lp + LP_B_O + 2u * col);
    wait_acc<kAr>(c, 3, 0);
    each_piece<NB>(O::slot(c, 3), [&](int k, const uint32_t (&acc)[16]) {
        uint32_t y[8];
        if (k > 0) bias = load_bias(lp + LP_B_O + 2u * col + 32 * k);
        descale16<false, Cfg<kAr>::kOutF16 ? kAccPlain : kAccInt>(acc, so.scale, sw, bias, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[8 * k + i] = as_u32(__hadd2(as_h2(x[8 * k + i]), as_h2(y[i])));
    });
}

// ---- FFN ----
// Chunk by chunk: ff1's epilogue (descale, bias, ReLU, row maximum), the meeting of the row's threads for the
// maximum, quantisation into the ff2 operand, which starts that chunk's ff2 product.  A chunk's epilogue
// comes before the quantisation of the one before it, so that nobody waits where they meet.  ff2's products
// run under the epilogues that follow; their four sums are added to the fp16 running total in order.
template <int NB, int kAr>
__device__ __forceinline__ void ffn_block(const Row& c, uint32_t lp, float sa, uint32_t (&x)[8 * NB]) {
    using O = Own<NB>;
    const int col = O::col(c), row = O::row(c);
    float s1[4];
    uint32_t hid[2][8 * NB];
    const uint32_t maxima = c.smem + SM_MAX + 256u + 4u * row;
    auto epilogue = [&](int ch, uint32_t (&h)[8 * NB]) {
        const uint32_t bias_at = lp + LP_B_FF1 + 2u * (256 * ch + col);
        const float sw = lds_f(lp + LP_SW_FF1 + 4u * (2 * ch + (col >> 7)));
        Bias bias = load_bias(bias_at);
        wait_acc<kAr>(c, ch, 1);
        each_piece<NB>(O::slot(c, ch), [&](int i, const uint32_t (&acc)[16]) {
            if (i > 0) bias = load_bias(bias_at + 32 * i);
            descale16<true, kAr == kArE4M3 ? kAccFloat : kAccInt>(acc, sa, sw, bias, &h[8 * i]);
        });
        max_to(maxima + 256u * ch, amax_h2<8 * NB>(h, false), c, ch);
    };
    epilogue(0, hid[0]);
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        if (ch < 3) epilogue(ch + 1, hid[(ch + 1) & 1]);
        board_sync<NB>(c, ch);
        const float amax = lds_f(maxima + 256u * ch);
        const Scale sc = kAr == kArE4M3 ? scale_e4m3(amax) : scale_u8(amax);
        s1[ch] = sc.scale;
#pragma unroll
        for (int i = 0; i < NB; ++i)
            store_operand8<NB, kAr == kArE4M3>(c, c.h + ch * 2 * O::kSlab, i, &hid[ch & 1][8 * i], sc.inverse);
        publish(c, B_H + ch);
    }
    uint32_t run[8 * NB];
#pragma unroll
    for (int i = 0; i < 8 * NB; ++i) run[i] = 0u;
    const float s2 = lds_f(lp + LP_SW_FF2 + 4u * (col >> 7));
    const uint64_t s2_2 = pk2(s2, s2);
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        wait_acc<kAr>(c, ch, 2);
        const uint64_t s1_2 = pk2(s1[ch], s1[ch]);
        each_piece<NB>(O::slot(c, ch), [&](int k, const uint32_t (&acc)[16]) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                // `float(acc) * sa * sw + float(run)`: the second product and the sum are one fma (and
                // with the zero that the total starts from, a plain product)
                const uint64_t f = mul2(kAr == kArE4M3 ? pk2(__uint_as_float(acc[2 * i]), __uint_as_float(acc[2 * i + 1]))
                                                       : pk2(static_cast<float>(static_cast<int>(acc[2 * i])),
                                                             static_cast<float>(static_cast<int>(acc[2 * i + 1]))), s1_2);
                run[8 * k + i] = f2_to_h2(fma2(f, s2_2, h2_to_f2(run[8 * k + i])));
            }
        });
    }
    // + b_ff2, residual: x = fp16(x + fp16(run + b))
#pragma unroll
    for (int v = 0; v < 2 * NB; ++v) {
        const uint4 bv = lds128(lp + LP_B_FF2 + 2u * col + 16u * v);
        const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * v + k;
            x[i] = as_u32(__hadd2(as_h2(x[i]), __hadd2(as_h2(run[i]), as_h2(bw[k]))));
        }
    }
}

// The fp16 arithmetic's FFN: ff1's epilogue is bias and ReLU, a chunk goes out as ff2's fp16 operand, and
// ff2's fp16 accumulators (slot 0) run on through the four chunks.  H holds two chunks, so the third and the fourth
// are written when ff2 is done with the first and the second (completions of slots 0 and 1 that say no more than
// that); a completion of slot 2 says that the sums are there.  The products follow one another in the order ff1 0, 1,
// ff2 0, ff1 2, ff2 1, ff1 3, ff2 2, 3: each has its operand when its turn comes, and a chunk's place is free when
// the chunk is (all of ff1 first, and two chunks to an arrival: 1,000 cycles of a two-board layer's 23,400 more).
template <int NB>
__device__ __forceinline__ void ffn_block_f16(const Row& c, uint32_t lp, uint32_t (&x)[8 * NB]) {
    using O = Own<NB>;
    const int col = O::col(c);
#pragma unroll 1
    for (int ch = 0; ch < 4; ++ch) {
        const uint32_t bias_at = lp + LP_B_FF1 + 2u * (256 * ch + col);
        Bias bias = load_bias(bias_at);
        wait_acc<kArF16>(c, ch, 1);
        if (ch >= 2) wait_acc<kArF16>(c, ch - 2, 2);
        each_piece<NB>(O::slot(c, ch), [&](int i, const uint32_t (&acc)[16]) {
            uint32_t h[8];
            if (i > 0) bias = load_bias(bias_at + 32 * i);
            descale16<true, kAccPlain>(acc, 1.f, 1.f, bias, h);
            store_operand16<NB>(c, c.h + (ch & 1) * 4 * O::kSlab, i, h);
        });
        publish(c, B_H + ch);
    }
    Bias bias = load_bias(lp + LP_B_FF2 + 2u * col);
    wait_acc<kArF16>(c, 2, 2);
    each_piece<NB>(O::slot(c, 0), [&](int k, const uint32_t (&acc)[16]) {
        uint32_t y[8];
        if (k > 0) bias = load_bias(lp + LP_B_FF2 + 2u * col + 32 * k);
        descale16<false, kAccPlain>(acc, 1.f, 1.f, bias, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[8 * k + i] = as_u32(__hadd2(as_h2(x[8 * k + i]), as_h2(y[i])));
    });
}

// ---- heads ----
// The "prenorm" value head (see `prenorm_value`, whose order of sums this keeps): the column means over the
// board's live tokens go into the board's list buffer, which the expansion warp touches only once this
// tile's logits are staged.
template <int NB>
__device__ __forceinline__ void prenorm_means(const Row& c, uint32_t alive, const uint32_t (&x)[8 * NB]) {
    using O = Own<NB>;
    const bool live = (alive >> c.lane) & 1u;
    const int nlive = __popc(alive);
    const float inv_live = 1.0f / static_cast<float>(nlive > 0 ? nlive : 1);
    float2 mine = make_float2(0.f, 0.f);                     // lane i keeps column pair i
#pragma unroll
    for (int i = 0; i < 8 * NB; ++i) {
        const float2 f = __half22float2(as_h2(x[i]));
        float a0 = live ? f.x : 0.f, a1 = live ? f.y : 0.f;
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, off);
            a1 += __shfl_xor_sync(0xffffffffu, a1, off);
        }
        if (c.lane == i) mine = make_float2(__fmul_rn(a0, inv_live), __fmul_rn(a1, inv_live));
    }
    if (c.lane < 8 * NB) {
        const uint32_t at = c.smem + SM_LIST + kListBytes * O::board(c) + 4u * O::col(c) + 8u * c.lane;
        sts32(at, __float_as_uint(mine.x));
        sts32(at + 4u, __float_as_uint(mine.y));
    }
}
// The three logits, in one warp, while the head product runs: lane & 3 is the quarter of the columns
// (32 q .. + 31 and 128 + 32 q .. + 31), lane >> 2 the sum: of the means, of their squares, of
// means x gamma x value row k (with it gamma x value row k), of beta x value row k.  Out of line: inlined, this
// head's code slows the networks that do not have it (4096 positions on tiles of one SM, int8 1690 us against 1675, with
// edge lists 1748 against 1727).
template <int NB>
__device__ __noinline__ void prenorm_logits(const Row& c, const Params& p, float (&logit)[3]) {
    const uint32_t means = c.smem + SM_LIST + kListBytes * Own<NB>::board(c);
    const int quarter = c.lane & 3, kind = c.lane >> 2, k = kind < 2 ? 0 : (kind - 2) % 3;
    float t = 0.f, t2 = 0.f;
#pragma unroll 1
    for (int i = 0; i < 32; ++i) {
        const int col = 128 * (i >> 4) + 32 * quarter + 2 * (i & 15);
        const float2 a = make_float2(lds_f(means + 4u * col), lds_f(means + 4u * col + 4u));
        const float2 g = __half22float2(as_h2(__ldg(reinterpret_cast<const uint32_t*>(p.tail + col))));
        const float2 b = __half22float2(as_h2(__ldg(reinterpret_cast<const uint32_t*>(p.tail + kD + col))));
        const float2 w = __half22float2(as_h2(__ldg(reinterpret_cast<const uint32_t*>(p.tail + (2 + k) * kD + col))));
        const float2 u = kind < 2 ? a : kind < 5 ? make_float2(__fmul_rn(a.x, g.x), __fmul_rn(a.y, g.y)) : b;
        t = prenorm_add(t, u, kind == 0 ? make_float2(1.f, 1.f) : kind == 1 ? a : w);
        t2 = prenorm_add(t2, g, w);
    }
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
        t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, off));
        t2 = __fadd_rn(t2, __shfl_xor_sync(0xffffffffu, t2, off));
    }
    const float tot = __shfl_sync(0xffffffffu, t, 0), totq = __shfl_sync(0xffffffffu, t, 4);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        logit[i] = prenorm_logit(tot, totq, __shfl_sync(0xffffffffu, t, 8 + 4 * i), __shfl_sync(0xffffffffu, t2, 8 + 4 * i),
                                 __shfl_sync(0xffffffffu, t, 20 + 4 * i), p.eps);
}

// Final norm into the head product's fp16 operand, then the epilogue: the product's 128 output columns
// (64 policy, 4 promotion, value, padding) lie 8 NB to a thread.  Policy columns are masked and stored
// by the threads that hold them; with a fused expansion the logits are staged for the expansion warps.
template <int NB, int kAr, bool kExpand>
__device__ __forceinline__ void heads(const Row& c, const Params& p, int board, bool valid, int ctl, uint32_t alive,
                                      const uint32_t (&x)[8 * NB]) {
    using O = Own<NB>;
    const int col = O::col(c), row = O::row(c), lane = c.lane;
    const long grow = static_cast<long>(board) * kT + lane;
    if (p.vmode == 2) prenorm_means<NB>(c, alive, x);         // (the norm's meetings make them everybody's)
    {
        const float4 st = row_statistics<NB, kAr>(c, p, x);
        const uint64_t nmean2 = pk2(st.x, st.x), rstd2 = pk2(st.y, st.y);
        const uint4* g4 = reinterpret_cast<const uint4*>(p.tail + col);
        const uint4* b4 = reinterpret_cast<const uint4*>(p.tail + kD + col);
#pragma unroll
        for (int v = 0; v < 2 * NB; ++v) {
            const uint4 gv = __ldg(g4 + v), bv = __ldg(b4 + v);
            const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, bw[4] = {bv.x, bv.y, bv.z, bv.w};
            uint32_t y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                y[j] = f2_to_h2(fma2(mul2(add2(h2_to_f2(x[4 * v + j]), nmean2), rstd2), h2_to_f2(gw[j]), h2_to_f2(bw[j])));
            store_operand<NB>(c.h + kHeadA + (col >> 6) * O::kSlab + sw_off(row, ((col & 63) >> 3) + v), make_uint4(y[0], y[1], y[2], y[3]));
        }
        publish(c, B_A);
    }
    // output columns of this thread: hc .. hc + 8 NB - 1
    const int within = 16 * c.s + (NB == 1 ? 8 * (c.q & 1) : 0), hc = 64 * (c.q >> 1) + within;
    // while the product runs: the legality words
    unsigned long long lw = ~0ull;
    if (p.legal != nullptr && p.policy != nullptr && valid && hc < 64) lw = p.legal[grow];
    float pre[3] = {0.f, 0.f, 0.f};
    if (p.vmode == 2 && hc == 64) prenorm_logits<NB>(c, p, pre);
    wait_acc<kAr>(c, 0, 0);
    uint32_t v[4 * NB];
    {
        uint32_t acc[8 * NB];
        const uint32_t t = c.tm + within;
        if constexpr (NB == 1) tmem_ld8(t, acc); else tmem_ld16(t, acc);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 4 * NB; ++i) v[i] = __byte_perm(acc[2 * i], acc[2 * i + 1], 0x5410);
    }
    if constexpr (kExpand) {
        if (hc < 64) {
#pragma unroll
            for (int k = 0; k < NB; ++k)
                sts128(c.h + kStagePolicy + 4096u * O::board(c) + sw_off(lane, (hc >> 3) + k),
                       make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]));
        } else if (hc == 64) {
            sts128(c.h + kStageAux + 512u * O::board(c) + 16u * lane, make_uint4(v[0], v[1], v[2], v[3]));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(c.smem, B_STAGED));
    }
    if (hc < 64) {
        if (valid && p.policy != nullptr) {
            const uint32_t bits = static_cast<uint32_t>(lw >> hc);
#pragma unroll
            for (int i = 0; i < 4 * NB; ++i) {
                if (!((bits >> (2 * i)) & 1u)) v[i] = (v[i] & 0xffff0000u) | 0xfc00u;
                if (!((bits >> (2 * i + 1)) & 1u)) v[i] = (v[i] & 0x0000ffffu) | 0xfc000000u;
            }
            store_words<4 * NB>(p.policy + grow * 64 + hc, v);
        }
    } else if (hc == 64) {
        if (valid && p.promo != nullptr) *reinterpret_cast<uint2*>(p.promo + grow * 4) = make_uint2(v[0], v[1]);
        // value logits: columns 68, 69, 70
        float a = __low2float(as_h2(v[2])), b = __high2float(as_h2(v[2])), d = __low2float(as_h2(v[3]));
        if (p.vmode == 1) {
            // live tokens in slot order, one after the other
            float ta = 0.f, tb = 0.f, td = 0.f;
#pragma unroll 1
            for (int tt = 0; tt < kT; ++tt) {
                const float at = __shfl_sync(0xffffffffu, a, tt), bt = __shfl_sync(0xffffffffu, b, tt);
                const float dt = __shfl_sync(0xffffffffu, d, tt);
                if ((alive >> tt) & 1u) { ta += at; tb += bt; td += dt; }
            }
            const int nlive = __popc(alive);
            const float inv = 1.0f / static_cast<float>(nlive > 0 ? nlive : 1);
            a = ta * inv; b = tb * inv; d = td * inv;
        }
        if (p.vmode == 2) { a = pre[0]; b = pre[1]; d = pre[2]; }
        const bool writer = p.vmode != 0 ? lane == 0 : lane == (ctl < 0 ? 31 : 15);
        if (writer && valid && p.value != nullptr) {
            float o;
            if (p.n_value == 1) {
                o = tanhf(a);
            } else {
                const float m = fmaxf(a, fmaxf(b, d));
                const float ea = expf(a - m), eb = expf(b - m), ec = expf(d - m);
                o = (ec - ea) / (ea + eb + ec);
            }
            if (p.vmode != 0 && ctl < 0) o = -o;
            p.value[board] = o;
        }
    }
}

// The fused expansion has two warps of its own, one per board of a tile: they make the legal words
// while the layers run and expand while the next tile begins.  4096 positions on tiles of one SM: 1743 us with the words given
// and 1766 with the moves generated, where row warps between the head product and the next tile took 1793 and 1839; by
// pairs of SMs 1591 and 1595.  Where the rows' first FFN of the next tile would overwrite the staged logits they
// wait for B_EXPANDED.
template <int NB>
__device__ __forceinline__ void expander(uint32_t smem, uint8_t* smem_gen, uint32_t h, volatile int* abort_flag, const Params& p,
                                         const Tiles<NB>& tiles, int which, int lane) {
    for (int k = 0; k < tiles.count(); ++k) {
        const int item = tiles.at(k) + which;
        const bool valid = which < NB && item < tiles.n;
        int board = item, ctl = 1;
        uint32_t word = 0u;
        unsigned long long moves = 0ull;
        if (valid) {
            if (p.leaf_index != nullptr) board = p.leaf_index[item];
            const long at = static_cast<long>(board) * kT + lane;
            word = p.boards[at];
            ctl = static_cast<int>(p.control[board]);
            bool in_check;
            moves = p.legal != nullptr ? p.legal[at] : bfmg::legal_word(word, ctl, in_check);
        }
        mbar_wait<200>(bar(smem, B_STAGED), k & 1u, abort_flag, kErrRowAcc);
        __syncwarp();
        if (valid)
            expand_board(p, board, lane, true, word, ctl, moves, h + kStagePolicy + 4096u * which + 128u * lane, lane & 7,
                         h + kStageAux + 512u * which + 16u * lane, smem_gen + SM_LIST + kListBytes * which);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(smem, B_EXPANDED));
    }
}

// Where 16-byte piece `part` of a token's columns lies in a warp's block: `kLanes` pieces to a token, moved so that
// eight tokens' same piece, and what eight lanes next to each other hold, hit all banks.
template <int kLanes>
__device__ __forceinline__ uint32_t embed_off(int token, int part) {
    return 16u * (kLanes * token + (part ^ ((token / (8 / kLanes)) & (kLanes - 1))));
}

// One tile of NB boards, from the piece words to the outputs.
template <int NB, int kAr, bool kExpand>
__device__ __forceinline__ void row_tile(Row& c, const Params& p, int first) {
    using O = Own<NB>;
    const int item = first + O::board(c), lane = c.lane, col = O::col(c);
    const bool valid = item < c.n;
    const int board = (valid && p.leaf_index != nullptr) ? p.leaf_index[item] : item;
    const uint32_t word = valid ? p.boards[static_cast<long>(board) * kT + lane] : 0u;
    uint32_t alive = __ballot_sync(0xffffffffu, ((word >> 11) & 1u) == 0u);
    const int ctl = valid ? static_cast<int>(p.control[board]) : 1;
    if (!valid) alive = 0xffffffffu;
    uint32_t x[8 * NB];
    // ---- embedding: ((square + type_special) + color_turn) + (clock + rep), fp16 ----
    {
        const int stm = ctl < 0;
        const int clk = min(max((ctl < 0 ? -ctl : ctl) - 1, 0), kNClock - 1);
        const int rp = min(valid ? static_cast<int>(p.rep[board]) : 0, kNRep - 1);
        const int sq = word & 63;
        const int ts = min(static_cast<int>(((word >> 6) & 7) * 2 + ((word >> 9) & 1)), kNTypeSpecial - 1);
        const int ct = ((word >> 10) & 1) * 2 + stm;
        // A token's columns of the three tables that go by token are read by 2 NB lanes next to each other, 16 bytes to a
        // lane, summed there, and go to the token's own lane through the warp's 1 KB of the last tile's head operand
        // (32 / NB tokens at a time).  With every lane reading its own token's a warp's load touches 32 lines, one a cycle:
        // 1 % of a two-board tile more.
        constexpr int kLanes = 2 * NB, kTokens = 32 / kLanes;
        const int part = lane & (kLanes - 1);
        const int rows = (EMB_SQUARE + sq) | (EMB_TS + ts) << 8 | (EMB_CT + ct) << 16;
        constexpr int kAtOnce = 32 / NB;
        const uint32_t block = c.h + kHeadA + 1024u * (4 * c.q + c.s);
        const __half* emb = p.emb + col + 8 * part;
        const uint4 e = __ldg(reinterpret_cast<const uint4*>(emb + (EMB_CLOCK + clk) * kD));
        const uint4 f = __ldg(reinterpret_cast<const uint4*>(emb + (EMB_REP + rp) * kD));
        const uint32_t ew[4] = {e.x, e.y, e.z, e.w}, fw[4] = {f.x, f.y, f.z, f.w};
        uint4 a[kLanes], b[kLanes], d[kLanes];
#pragma unroll
        for (int k = 0; k < kLanes; ++k) {
            const int r = __shfl_sync(0xffffffffu, rows, kTokens * k + lane / kLanes);
            a[k] = __ldg(reinterpret_cast<const uint4*>(emb + (r & 255) * kD));
            b[k] = __ldg(reinterpret_cast<const uint4*>(emb + ((r >> 8) & 255) * kD));
            d[k] = __ldg(reinterpret_cast<const uint4*>(emb + (r >> 16) * kD));
        }
#pragma unroll
        for (int pass = 0; pass < NB; ++pass) {
#pragma unroll
            for (int k = 2 * pass; k < 2 * pass + 2; ++k) {
                const uint32_t aw[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, bw[4] = {b[k].x, b[k].y, b[k].z, b[k].w};
                const uint32_t dw[4] = {d[k].x, d[k].y, d[k].z, d[k].w};
                uint32_t y[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __half2 v = __hadd2(as_h2(aw[j]), as_h2(bw[j]));
                    v = __hadd2(v, as_h2(dw[j]));
                    y[j] = as_u32(__hadd2(v, __hadd2(as_h2(ew[j]), as_h2(fw[j]))));
                }
                sts128(block + embed_off<kLanes>((kTokens * k + lane / kLanes) & (kAtOnce - 1), part), make_uint4(y[0], y[1], y[2], y[3]));
            }
            __syncwarp();
            if (lane / kAtOnce == pass) {
#pragma unroll
                for (int k = 0; k < kLanes; ++k) {
                    const uint4 v = lds128(block + embed_off<kLanes>(lane & (kAtOnce - 1), k));
                    x[4 * k] = v.x; x[4 * k + 1] = v.y; x[4 * k + 2] = v.z; x[4 * k + 3] = v.w;
                }
            }
            __syncwarp();
        }
    }
    const int id = 128 * c.q + 32 * c.s + lane;              // 0 .. 511
    // half-layers, so that the norm's code is there once
    const int n_half = 2 * p.n_layers;
#pragma unroll 1
    for (int half = 0; half < n_half; ++half) {
        const uint32_t lp = layer_params(c);
        if ((half & 1) == 0) wait_params(c);
        // the row maxima start at zero: the hidden chunks' are cleared before the attention norm's
        // meetings, the attention output's before the FFN norm's (and at the start), ahead of their use
        const uint32_t mx = c.smem + SM_MAX + 4u * O::row(c);
        if ((half & 1) == 0 && O::member(c) < 4) sts32(mx + 256u * (1 + O::member(c)), 0u);
        if (((half & 1) || half == 0) && O::member(c) == 4) sts32(mx, 0u);
        const float sa = norm_to_operand<NB, kAr>(c, p, x, kAr == kArF16 || (half & 1) == 0);
        if ((half & 1) == 0) {
            attention_block<NB, kAr>(c, lp, sa, alive, x);
        } else {
            if (kExpand && half == 1 && c.tiles != 0) {
                mbar_wait(bar(c.smem, B_EXPANDED), (c.tiles - 1u) & 1u, c.abort_flag, kErrRowAcc);
                __syncwarp();
            }
            if constexpr (kAr == kArF16) ffn_block_f16<NB>(c, lp, x);
            else ffn_block<NB, kAr>(c, lp, sa, x);
            c.layers++;
        }
    }
    if (id < static_cast<int>(kTailBytes / 128)) prefetch_l1(reinterpret_cast<const uint8_t*>(p.tail) + 128 * id);
    heads<NB, kAr, kExpand>(c, p, board, valid, ctl, alive, x);
    c.tiles++;
}

// ---- weight stream ----
// Of `sent` stages the last ones' consumption, which no further stage is sent for, arrives too, from the first SM's
// products at both SMs' barriers: waited for, so that no arrival is on its way when the next grid has its own barriers
// here.  (Once a launch, beside the heads: 0.3 us of a batch of 1 (81.0), 5 us of 4096 (1538).)
template <uint32_t kStages>
__device__ __forceinline__ void drain(uint32_t smem, volatile int* abort_flag, uint32_t sent) {
#pragma unroll 1
    for (uint32_t i = sent > kStages ? sent - kStages : 0u; i < sent; ++i)
        mbar_wait(bar(smem, B_EMPTY + i % kStages), (i / kStages) & 1u, abort_flag, kErrProducer);
}
// The blob's stages are the four-board kernel's: per head pair [Q 64 | K 64 | V 64 rows], then 128-row
// units, two to each 256-row product.  A stage here is 256 rows of one K-slab, put together from four
// or two of their pieces.  The whole warp walks the stages and waits; one elected lane issues.
// Each SM of the pair loads its half of every product's rows: the first or the second of two units, two of four head pairs.
template <int kAr>
__device__ __forceinline__ void producer(uint32_t smem, volatile int* abort_flag, const Params& p, int n_tiles, uint32_t rank) {
    using C = Cfg<kAr>;
    constexpr uint32_t kStages = Map<kAr>::kStages, kRing = Map<kAr>::SM_RING;
    uint32_t i = 0;
    // the next stage: `copies(dst, barrier)` of `bytes` in all
    auto stage = [&](uint32_t bytes, auto&& copies) {
        const uint32_t k = i % kStages;
        if (i == kStages && !p.after_waves) { previous_grid_wait(); next_grid_may_start(); }   // (before the first wait that has a limit)
        if (i >= kStages) mbar_wait(bar(smem, B_EMPTY + k), (i / kStages - 1u) & 1u, abort_flag, kErrProducer);
        if (elect_one()) {
            mbar_arrive_expect_tx(bar(smem, B_FULL + k), bytes);
            copies(smem + kRing + k * kStage, bar(smem, B_FULL + k));
        }
        ++i;
    };
    // K-slab s of the product whose two 128-row units start at `u0` and `u1`
    auto two_units = [&](const uint8_t* u0, const uint8_t* u1, int s) {
        stage(kStage, [&](uint32_t dst, uint32_t full) { bulk_g2s(dst, (rank ? u1 : u0) + s * kRStage, kRStage, full); });
    };
    // The scales and biases of a layer go into one of two places.  Those of the next layer are sent when
    // the ring has taken as many of this layer's stages as it holds and one more: Q's first has then been
    // consumed, so every row warp has published this layer's first operand and is done with the layer before,
    // whose place they take.
    uint32_t g = 0;             // layers whose parameters have been sent
    auto params = [&](int layer) {
        if (elect_one()) {
            const uint32_t full = bar(smem, B_PAR + (g & 1u));
            mbar_arrive_expect_tx(full, kLparamStride);
            bulk_g2s(smem + SM_PAR + (g & 1u) * kLparamStride, p.lparams + static_cast<size_t>(layer) * kLparamStride, kLparamStride, full);
        }
        ++g;
    };
    if (n_tiles > 0) params(0);
    for (int tile = 0; tile < n_tiles; ++tile) {
        const uint8_t* src = p.wstream;
        for (int layer = 0; layer < p.n_layers; ++layer, src += C::kLayerStream) {
            const uint32_t begin = i;
            // (an FFN stage: the ring is no deeper than the stages before the FFN and ff1's)
            constexpr uint32_t kBefore = 3 * C::kQkvSlabs + C::kOutSlabs, kFirstFfn = kBefore > kStages ? kBefore : kStages;
            static_assert(kFirstFfn < kBefore + 8 * C::kFfnSlabs, "the parameters are sent within the layer");
            for (int m = 0; m < 3; ++m)                                     // Q, K, V
                for (int s = 0; s < C::kQkvSlabs; ++s)
                    stage(kStage, [&](uint32_t dst, uint32_t full) {
                        const uint8_t* from = src + s * kQStage + m * 8192 + 2 * rank * C::kQkvSlabs * kQStage;
#pragma unroll
                        for (int j = 0; j < 2; ++j) bulk_g2s(dst + 8192 * j, from + C::kQkvSlabs * j * kQStage, 8192, full);
                    });
            const uint8_t* out = src + 4 * C::kQkvSlabs * kQStage;
            for (int s = 0; s < C::kOutSlabs; ++s) two_units(out, out + C::kOutSlabs * kRStage, s);
            // ff1 chunks 0-3, then ff2 chunks 0-3 (fp16: see `ffn_block_f16`); where their two units lie in the packed order
            const uint8_t* ffn = out + 2 * C::kOutSlabs * kRStage;
            for (int k = 0; k < 8; ++k) {
                int u0, u1;
                if (kAr == kArF16) {
                    const int u = (0x76352410u >> (4 * k)) & 7, ch = u & 3;
                    u0 = u < 4 ? (ch == 0 ? 0 : 4 * ch - 2) : (ch < 3 ? 4 * ch + 3 : 14);
                    u1 = u < 4 ? 4 * ch + 1 : (ch < 3 ? 4 * ch + 4 : 15);
                } else {
                    u0 = (0xEC84A620u >> (4 * k)) & 15u;
                    u1 = u0 + 1;
                }
                for (int s = 0; s < C::kFfnSlabs; ++s) {
                    two_units(ffn + u0 * C::kFfnSlabs * kRStage, ffn + u1 * C::kFfnSlabs * kRStage, s);
                    if (i - begin == kFirstFfn + 1u) {
                        if (layer + 1 < p.n_layers) params(layer + 1);
                        else if (tile + 1 < n_tiles) params(0);
                    }
                }
            }
        }
        // (the second SM has rows 64 to 95 of the head's; what else its half of the product reads is left from before,
        // and no output comes from it)
        const uint32_t skip = rank ? 8192u : 0u, bytes = rank ? kHeadStage - 8192u : 8192u;
        for (uint32_t st = 0; st < kHeadStages; ++st, src += kHeadStage)
            stage(bytes, [&](uint32_t dst, uint32_t full) { bulk_g2s(dst, src + skip, bytes, full); });
    }
    drain<kStages>(smem, abort_flag, i);
    // after a time-out copies may still be in flight: a bounded while for them to land
    if (*abort_flag != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) { }
    }
}

// ---- MMA issue ----
struct Issue {
    uint32_t smem, tmem;
    volatile int* abort_flag;
    uint32_t i, a, h;           // weight stages, A operands, hidden pairs consumed
};
// One product: `slabs` K-slabs of 128 bytes; `more`: on top of what the slot holds; `done`: the slot's
// barrier that its completion goes to (-1: none).  The whole warp walks the schedule and waits; one
// elected lane -- the same every time -- issues.  Stage by stage: waiting for two at once, which the four-board form gains from, costs 5 % of a one-board
// tile and 19 % of a two-board one in fp16, where the stages arrive no sooner than they are wanted.
template <int kAr, int kKind>
__device__ __forceinline__ void issue_unit(Issue& st, uint32_t d, uint32_t a_base, uint32_t slab, int slabs, uint32_t idesc,
                                           int done, bool more = false) {
    constexpr uint32_t kStages = Map<kAr>::kStages;
    for (int s = 0; s < slabs; ++s) {
        const uint32_t k = st.i % kStages;
        mbar_wait_cluster(bar(st.smem, B_FULL + k), (st.i / kStages) & 1u, st.abort_flag, kErrMmaWeights);
        tc_fence_after();
        if (elect_one()) {
            const uint64_t ad = umma_desc_k128(a_base + s * slab), bd = umma_desc_k128(st.smem + Map<kAr>::SM_RING + k * kStage);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const uint32_t accumulate = (more || (s | kk) != 0) ? 1u : 0u;
                if (kKind == kKindF16)     umma_pair_f16(d, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                else if (kKind == kKindF8) umma_pair_f8(d, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                else                       umma_pair_i8(d, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
            }
            tc_commit_pair(bar(st.smem, B_EMPTY + k));
            if (s == slabs - 1 && done >= 0) tc_commit_pair(bar(st.smem, B_ACC + done));
        }
        st.i++;
    }
}
// The pair's second SM issues nothing: its MMA warp tells the first which weights have arrived.
template <int kAr>
__device__ __forceinline__ void relay(uint32_t smem, volatile int* abort_flag, uint32_t stages) {
    constexpr uint32_t kStages = Map<kAr>::kStages;
    for (uint32_t i = 0; i < stages; ++i) {
        const uint32_t k = i % kStages;
        mbar_wait(bar(smem, B_FULL + k), (i / kStages) & 1u, abort_flag, kErrMmaWeights);
        if (elect_one()) mbar_arrive_first(bar(smem, B_FULL + k));
    }
}
__device__ __forceinline__ void issue_wait(const Issue& st, int b, uint32_t n) {
    mbar_wait_cluster(bar(st.smem, b), n & 1u, st.abort_flag, kErrMmaOperand);
    tc_fence_after();
}
template <int NB, int kAr>
__device__ __forceinline__ void issue_tile(Issue& st, int n_layers) {
    using O = Own<NB>;
    using C = Cfg<kAr>;
    constexpr uint32_t kM = 128;                             // 64 rows of each SM
    constexpr uint32_t kI_S8 = umma_idesc(kAccS32, kFmtS8, kFmtS8, kM, 256);
    constexpr uint32_t kI_F16 = umma_idesc(kAccF16, kFmtF16, kFmtF16, kM, 256);
    constexpr uint32_t kI_E4M3 = umma_idesc(kAccF32, kFmtE4M3, kFmtE4M3, kM, 256);
    constexpr uint32_t kI_QKV = C::kQkvF16 ? kI_F16 : kI_S8, kI_OUT = C::kOutF16 ? kI_F16 : kI_S8;
    constexpr uint32_t kI_FF1 = kAr == kArF16 ? kI_F16 : kAr == kArE4M3 ? kI_E4M3 : kI_S8;
    constexpr uint32_t kI_FF2 = kAr == kArF16 ? kI_F16 : kAr == kArE4M3 ? kI_E4M3
                                              : umma_idesc(kAccS32, kFmtU8, kFmtS8, kM, 256);
    constexpr uint32_t kI_HEAD = umma_idesc(kAccF16, kFmtF16, kFmtF16, kM, 128);
    constexpr int kQkvKind = C::kQkvF16 ? kKindF16 : kKindI8, kOutKind = C::kOutF16 ? kKindF16 : kKindI8;
    constexpr int kFfnKind = kAr == kArE4M3 ? kKindF8 : (kAr == kArF16 ? kKindF16 : kKindI8);
    const uint32_t a = st.smem + SM_A, h = st.smem + Map<kAr>::SM_H;
    for (int layer = 0; layer < n_layers; ++layer) {
        issue_wait(st, B_A, st.a++);
        for (int m = 0; m < 3; ++m)
            issue_unit<kAr, kQkvKind>(st, st.tmem + O::kSlot * m, a, O::kSlab, C::kQkvSlabs, kI_QKV, m);
        issue_wait(st, B_A, st.a++);
        issue_unit<kAr, kOutKind>(st, st.tmem + O::kSlot * 3, a, O::kSlab, C::kOutSlabs, kI_OUT, 3);
        issue_wait(st, B_A, st.a++);
        auto ff1 = [&](int ch) {
            issue_unit<kAr, kFfnKind>(st, st.tmem + O::kSlot * ch, a, O::kSlab, C::kFfnSlabs, kI_FF1, ch);
        };
        for (int ch = 0; ch < (kAr == kArF16 ? 2 : 4); ++ch) ff1(ch);
        for (int ch = 0; ch < 4; ++ch) {
            issue_wait(st, B_H + ch, st.h);
            if (kAr == kArF16) {
                issue_unit<kAr, kFfnKind>(st, st.tmem, h + (ch & 1) * 4 * O::kSlab, O::kSlab, C::kFfnSlabs, kI_FF2,
                                          ch < 2 ? ch : ch == 3 ? 2 : -1, ch > 0);
                if (ch < 2) ff1(ch + 2);
            } else {
                issue_unit<kAr, kFfnKind>(st, st.tmem + O::kSlot * ch, h + ch * 2 * O::kSlab, O::kSlab, C::kFfnSlabs, kI_FF2, ch);
            }
        }
        st.h++;
    }
    issue_wait(st, B_A, st.a++);
    issue_unit<kAr, kKindF16>(st, st.tmem, h + kHeadA, O::kSlab, kHeadStages, kI_HEAD, 0);
}

// launch bounds: 640 threads, so that a scheduler's five warps fit its registers (96 each)
template <int kAr, bool kExpand, int NB>
__global__ void __launch_bounds__(640, 1) encoder_ws_kernel(const Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t smem = smem_u32(sm);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + SM_MISC + 4);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + SM_MISC);
    if (threadIdx.x == 0) {
        // the operands come from both SMs' warps, and the first SM hears of its own weights and of the second's
        for (int i = 0; i < B_COUNT; ++i)
            mbar_init(bar(smem, i), i == B_EXPANDED        ? 2
                                    : i < B_EMPTY          ? 2 - rank
                                    : i >= B_A && i < B_MAX ? 2 * kRowWarps
                                    : i >= B_MAX           ? kRowWarps
                                                           : 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == kMmaWarp) tmem_alloc_pair(smem + SM_MISC, TM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // The grid before this one may still be running.  Only the producer goes on without it: the first weights are
    // nobody's output.  One-board tiles beside this call's own two-board ones start without waiting for that grid, and
    // wait for it at their own end.  Their inputs may be outputs of the grid before it.  That one has ended: the two-board grid
    // lets them start only after its own wait, so what it wrote is in L2; the fence drops what this SM's L1 may hold from
    // before; and inputs are read by plain loads alone (an `__ldg` or a `const __restrict__` could be served or
    // moved past the fence).
    if (p.after_waves) {
        __threadfence();
    } else if (warp != kProducerWarp || p.leaf_count != nullptr) {
        previous_grid_wait();
        next_grid_may_start();
    }
    int n_eval = p.n;
    if (p.leaf_count != nullptr) n_eval = min(max(*p.leaf_count, 0), p.n);
    const Tiles<NB> tiles(n_eval, p.wave_ctas, gridDim.x, blockIdx.x, p.one_most);
    const int n_tiles = tiles.count();
    if constexpr (NB == 2) {
        if (warp < kRowWarps) take_registers<kRowRegisters>();
        else give_registers<kHelperRegisters>();
    }
    if (warp < kRowWarps) {
        Row c;
        c.lane = lane; c.q = warp & 3; c.s = warp >> 2;
        c.smem = smem; c.smem_gen = sm; c.h = smem + Map<kAr>::SM_H;
        c.tm = tmem + (static_cast<uint32_t>(32 * c.q) << 16);
        c.abort_flag = abort_flag;
        c.one2 = pk2(p.one, p.one);
        c.layers = c.tiles = 0;
        c.n = n_eval;
        for (int k = 0; k < n_tiles; ++k) row_tile<NB, kAr, kExpand>(c, p, tiles.at(k));
    } else if (warp == kProducerWarp) {
        producer<kAr>(smem, abort_flag, p, n_tiles, rank);
    } else if (warp >= kExpandWarp) {
        if constexpr (kExpand) expander<NB>(smem, sm, smem + Map<kAr>::SM_H, abort_flag, p, tiles, warp - kExpandWarp, lane);
    } else if (rank != 0) {
        using C = Cfg<kAr>;
        relay<kAr>(smem, abort_flag, n_tiles * (p.n_layers * (3 * C::kQkvSlabs + C::kOutSlabs + 8 * C::kFfnSlabs) + kHeadStages));
    } else {
        Issue st = {smem, tmem, abort_flag, 0, 0, 0};
        for (int k = 0; k < n_tiles; ++k) issue_tile<NB, kAr>(st, p.n_layers);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    // (the products read both SMs' shared memory, and barriers are written from both)
    cluster_sync();
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc_pair(tmem, TM_COLS);
    if (threadIdx.x == 0 && *abort_flag != 0) atomicCAS(p.status, 0, *abort_flag);
    previous_grid_wait();
}

}  // namespace ws
}  // namespace bf
