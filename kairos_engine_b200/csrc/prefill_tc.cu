/* prefill_tc.cu — the prefill GEMMs of the MoE feed-forward layer on the 5th-generation tensor
 * cores (tcgen05.mma, weights and accumulators in tensor memory), sm_100a only.
 *
 * Replaces the reference's prefill matmul for Q4B tensors (gemm_w, CF:13488-13518 of
 * src/backends/cuda/cuda_forward.cu: dequantise the whole tensor to a scratch matrix, then
 * cuBLAS) and its expert-major loop (gather / GEMM / GELU split / GEMM / scatter, CF:8925-8965)
 * with one grouped kernel per GEMM that dequantises Q4B tiles on the fly.
 *
 * Arithmetic. The reference multiplies w = code * f16 scale (exact in fp32, CF:1452-1464) by fp32
 * activations. fp16 operands alone cannot hold that (a 4-bit code times an 11-bit scale needs 14
 * bits; an fp32 activation 24), so both operands are split into two fp16 terms,
 *     w = w_hi + w_lo  (exact: w_hi = fp16(code*scale), w_lo = fma(code, scale, -w_hi)),
 *     x = x_hi + x_lo  (x_hi = fp16(x), x_lo = fp16(x - x_hi); |x - x_hi - x_lo| <= 2^-22 |x|),
 * and D += w_hi*x_hi + w_lo*x_hi + w_hi*x_lo accumulates in fp32 in tensor memory (the dropped
 * w_lo*x_lo term is below 2^-22 relative). That is three MMAs per k-step.
 *
 * Tile: two blocks of 128 weight rows (the MMA's M, one TMEM lane per weight row) x up to NMAX
 * activation rows (its N, a multiple of 16), K in stages of 64.
 *   - The weights are the A operand and live in tensor memory: an unpack thread owns one weight
 *     row, which is one TMEM lane, and stores its fp16 hi/lo values there (tcgen05.st). The
 *     unpacked weights therefore cost no shared-memory bandwidth, neither the write nor the read
 *     by every MMA; only the activation tile is read from shared memory (64 B per clock at any N).
 *   - The activation rows are N, so a group pays for its rows rounded up to 16, not to 128: with a
 *     few rows per expert the GEMM is a stream of weights, and with 256 the padding is some percent.
 *   gate|up GEMM : a block is 64 gate rows and the 64 up rows of the same outputs, 16 + 16 to a
 *                  32-lane quadrant, so that g and u of an output sit 16 lanes apart in one warp: one
 *                  shuffle per two outputs, then gelu(g)*u, split into fp16 hi/lo for the next GEMM;
 *   down GEMM    : a block is 128 consecutive rows, fp32 out.
 * A last tile with at most one block of rows left does that block only.
 * Packed codes come in by TMA (256 weights of 256 rows a time, 128-byte swizzle: the unpack threads
 * read their row's pieces without bank conflicts), activations by TMA from row lists sorted by
 * expert. Inside every group of 8 k the order is 0,4,1,5,2,6,3,7 on BOTH operands (the natural
 * order of the nibble unpack), which a dot product does not see.
 * Warps: 0-7 epilogue (TMEM lane quadrant = warp % 4, block = warp / 4), 8-23 unpack (the same, in
 * two sets that take alternate stages), 24 and 25 MMA issue (one per block), 26 activation TMA, 27
 * code TMA and TMEM allocation. Every wait is bounded.
 * A CTA draws its tiles from a counter; the code warp announces them to the others through a ring.
 * What bounds it (Gemma geometry, one B200): with a few rows per expert the chain of a stage in an MMA
 * warp, ~740 cycles at 37 tokens (two polls at once, twelve MMAs and two commits 300, the loop), beside
 * the unpack, ~136 instructions of the half-rate fp16 and integer pipes per 2048 weights, whose warps
 * wait half their time for a stage to be free; with 48 and more rows the tensor time of the three terms
 * (12, 16 and 32 cycles an MMA at N = 16, 32 and 64: 768 of ~870 cycles a stage at 64), and in the end
 * the power limit. A layer of 37 / 717 / 4096 tokens: 0.60 / 0.85 / 2.40 ms with the weights in shared
 * memory and 128 rows a tile, 0.18 / 0.40 / 1.78 ms with this.
 */
#include <map>
#include "prefill_tc.cuh"
#include "tc_common.cuh"
#include "launch.cuh"

namespace {
using namespace sp_tc;

constexpr int kBK = 64, kNGran = 16, kNMax = 64;
constexpr int kEpiWarps = 8, kItems = 8;                                /* items: the ring in which a CTA announces its next tiles */
constexpr uint32_t kBoxRows = 64, kBoxBytes = 128 * kBoxRows;          /* codes: 128 B (256 weights) of 64 rows */
constexpr uint32_t kChunkBytes = 4 * kBoxBytes;                        /* the four boxes of a tile: 32 KB per 256 k */
/* 512 TMEM columns: 2 blocks x kAccBufs x NMAX of accumulators from column 0, then a ring of three stages of unpacked
 * weights, 128 columns each (2 blocks x 64 k x hi/lo). Registers: the epilogue empties the accumulators into registers at
 * once, before it computes, so setmaxnreg moves registers to it. Tiles of 96 and of 128 rows were measured too (fewer
 * unpacks, but more registers for the epilogue and a shorter ring): the same within 2% at 4096 tokens, slower below. */
template <int NMAX> struct Cfg {
    static constexpr int kSets = 2, kUnpWarps = 8 * kSets, kWarps = kEpiWarps + kUnpWarps + 4, kThreads = 32 * kWarps;
    static constexpr int kAccBufs = NMAX == 32 ? 2 : 1, kACol = 2 * NMAX * kAccBufs, kAStages = 3, kACols = 2 * kBK;
    static constexpr int kBStages = 4, kCStages = 4;
    static constexpr uint32_t kBHalf = NMAX * 128u, kBStage = 2 * kBHalf;
    static constexpr uint32_t kCOff = kBStages * kBStage, kBarOff = kCOff + kCStages * kChunkBytes, kItemOff = kBarOff + 448;
    static constexpr uint32_t kScaleOff = kItemOff + 32 * kItems, kSmem = kScaleOff + 3 * 16 * 32 * kUnpWarps + 1024;     /* + alignment slack */
    static constexpr int kLaunchRegs = 72, kEpiRegs = 96, kUnpRegs = 64, kMiscRegs = 48;
    static_assert(32 * (kEpiWarps * kEpiRegs + kUnpWarps * kUnpRegs + 4 * kMiscRegs) <= kThreads * kLaunchRegs, "register split exceeds what the block is launched with");
    static_assert(kACol + kACols * kAStages <= 512, "tensor memory");
};

struct TcSeg {                     /* one GEMM of a launch: the shared expert's or the routed experts' */
    const uint16_t *bs[2];         /* block scales of the tensor feeding the gate / up rows (plain: both the same) */
    long long group_rows;          /* rows per group (expert) in the tensor */
    int up_off;                    /* pair: row offset of the up rows inside the group (0 with a separate up tensor) */
    int rows;                      /* valid output rows (pair: per half) */
    const int *tiles;              /* {group, first row, valid rows} per activation tile */
    const int *n_tiles;
    int m_tiles;
    __half *out_hi, *out_lo;       /* pair: geglu output rows of `rows` columns, split + permuted */
    float *out_f; int out_stride; const int *rowmap;  /* plain: out_f[(rowmap ? rowmap[r] : r) * stride + j] */
};
struct TcArgs { TcSeg seg[2]; int nseg; int K[2]; int *ticket; int *status; };       /* ticket: tiles handed out beyond the first of each CTA; zero at launch */
struct TcMaps { CUtensorMap codes[2][2], act[2][kNMax / kNGran]; };    /* [segment][gate / up]; activation boxes of 16, 32, 48 and 64 rows, hi and lo */

constexpr uint32_t kNegateA = 1u << 13;                                /* instruction descriptor: A enters with its sign flipped */

__device__ __forceinline__ int kperm(int j) { return (j & ~7) | ((j & 3) << 1) | ((j >> 2) & 1); }   /* slot of k = j */

/* one Q4B block (32 weights, one f16 scale) -> 16 registers of hi and (LO) of NEGATED lo halves (the MMA negates them
 * back: a sign is free there, and one instruction per two weights here). The nibbles j and j + 4 of a word become two
 * halves with an exponent that makes the nibble's place count one: 1024 + n in bits 0-3, 64 + n in bits 4-7; the nibbles
 * of the upper byte are shifted down once. The unpack is bound by the half-rate fp16 and integer pipes, so what counts is
 * 5 integer and 12 fp16 instructions per word of 8 weights. */
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t mask, uint32_t flip) {          /* one LOP3: `flip` has to be a register for that */
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(d) : "r"(a), "r"(mask), "r"(flip));
    return d;
}
__device__ __forceinline__ uint32_t in_register(uint32_t v) { uint32_t r; asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v)); return r; }
template <bool LO>
__device__ __forceinline__ void unpack_words(uint32_t w0, uint32_t w1, __half2 s2, uint32_t m1032, uint32_t m72, uint32_t t_hi, uint32_t t_lo) {
    const __half2 k1032 = __half2half2(__ushort_as_half((unsigned short)0x6408)), k72 = __half2half2(__ushort_as_half((unsigned short)0x5480));
    const __half2 ns2 = __hneg2(s2);
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const uint32_t w = q ? w1 : w0, up = w >> 8;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t x = j < 2 ? w : up;                                         /* code + 8 = the nibble with its top bit flipped */
            const uint32_t bits = j & 1 ? and_xor(x, 0x00F000F0u, m72) : and_xor(x, 0x000F000Fu, m1032);
            const __half2 c = __hsub2(*reinterpret_cast<const __half2 *>(&bits), j & 1 ? k72 : k1032);
            const __half2 h = __hmul2(c, s2);
            hi[4 * q + j] = *reinterpret_cast<const uint32_t *>(&h);
            if (LO) { const __half2 l = __hfma2(c, ns2, h); lo[4 * q + j] = *reinterpret_cast<const uint32_t *>(&l); }
        }
    }
    tmem_st8(t_hi, hi);
    if (LO) tmem_st8(t_lo, lo);
}
/* one Q4B block -> 16 columns of hi and of negated lo halves of this thread's TMEM lane */
template <bool LO>
__device__ __forceinline__ void unpack_block(const int4 &w, unsigned short scale, uint32_t m1032, uint32_t m72, uint32_t t_hi, uint32_t t_lo) {
    const __half2 s2 = __half2half2(__ushort_as_half(scale));
    unpack_words<LO>((uint32_t)w.x, (uint32_t)w.y, s2, m1032, m72, t_hi, t_lo);
    unpack_words<LO>((uint32_t)w.z, (uint32_t)w.w, s2, m1032, m72, t_hi + 8u, t_lo + 8u);
}

/* TERMS: 3 = all of w_hi*x_hi + w_lo*x_hi + w_hi*x_lo (exact to 2^-22); 2 = the weight rounded to fp16
 * (w_hi*x_hi + w_hi*x_lo); 1 = fp16 x fp16, the reference's SP_G4_GEMM_F16 mode (CF:13350-13365). */
struct __align__(16) Item { int sg, mt, grp, row0, nv, n16, nblk, KB; };      /* rows [row0, row0 + nv) of group grp x weight tile mt; KB 0: no more */

template <bool PAIR, int TERMS, int NMAX>
__global__ void __launch_bounds__(Cfg<NMAX>::kThreads, 1) k_tc_gemm(const __grid_constant__ TcArgs a, const __grid_constant__ TcMaps maps) {
    using C = Cfg<NMAX>;
    constexpr int BLK = PAIR ? 64 : 128;                                /* output rows of one block */
    constexpr int kMma = kEpiWarps + C::kUnpWarps, kActs = kMma + 2, kCodes = kMma + 3;      /* single warps: MMA issue (one per block), TMA */
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    /* a broadcast makes the warp number uniform to the compiler: what follows from it (roles, addresses, barriers) takes scalar
     * instructions and branches (gate|up launch of 37 tokens: 25.2 -> 19.8 M vector-integer instructions, 130 -> 126 us) */
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t bar0 = sbase + C::kBarOff;
    auto bfull = [&](int s) { return bar0 + 8u * s; };                  /* activation stages */
    auto bempty = [&](int s) { return bar0 + 32u + 8u * s; };
    auto cfull = [&](int s) { return bar0 + 64u + 8u * s; };            /* chunks of codes */
    auto cempty = [&](int s) { return bar0 + 96u + 8u * s; };
    auto afull = [&](int s, int blk) { return bar0 + 128u + 8u * (2 * s + blk); };      /* unpacked weights in TMEM: the two blocks keep apart rings, */
    auto aempty = [&](int s, int blk) { return bar0 + 176u + 8u * (2 * s + blk); };
    auto tfull = [&](int b, int blk) { return bar0 + 224u + 8u * (2 * b + blk); };      /* and apart accumulators */
    auto tempty = [&](int b, int blk) { return bar0 + 256u + 8u * (2 * b + blk); };
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + C::kBarOff + 288);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + C::kBarOff + 292);
    auto ifull = [&](int i) { return bar0 + 320u + 8u * (i % kItems); };                  /* items announced, and read by every other warp */
    auto iempty = [&](int i) { return bar0 + 384u + 8u * (i % kItems); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kBStages; s++) { mbar_init(bfull(s), 1); mbar_init(bempty(s), 2); }
        for (int s = 0; s < C::kCStages; s++) { mbar_init(cfull(s), 1); mbar_init(cempty(s), C::kUnpWarps); }
        for (int blk = 0; blk < 2; blk++) {
            for (int s = 0; s < C::kAStages; s++) { mbar_init(afull(s, blk), 4); mbar_init(aempty(s, blk), 1); }
            for (int b = 0; b < 2; b++) { mbar_init(tfull(b, blk), 1); mbar_init(tempty(b, blk), kEpiWarps / 2); }
        }
        for (int i = 0; i < kItems; i++) { mbar_init(ifull(i), 1); mbar_init(iempty(i), C::kWarps - 1); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kCodes) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void *)tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    sp_pdl_wait();
    sp_pdl_next();

    Item *items = reinterpret_cast<Item *>(smem + C::kItemOff);
    bool failed = false;
    /* the CTA's i-th tile, for every warp but the one that announces it */
    auto announced = [&](int i) { return mbar_wait(ifull(i), (uint32_t)(i / kItems) & 1u, abort_flag); };
    auto read = [&](int i) { __syncwarp(); mbar_arrive_lane0(iempty(i), lane); };

    if (warp < kEpiWarps) {
        /* ---------------- epilogue: TMEM -> registers, the accumulators are free again, then -> global */
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kEpiRegs));
        const int quad = warp & 3, blk = warp >> 2;
        int lt = 0;
        for (int i = 0;; i++) {
            if (!announced(i)) { failed = true; break; }
            const Item t = items[i % kItems];
            read(i);
            if (t.KB == 0) break;
            if (blk >= t.nblk) continue;
            const TcSeg &s = a.seg[t.sg];
            const int b = lt % C::kAccBufs; const uint32_t ph = (lt / C::kAccBufs) & 1;
            lt++;
            if (!mbar_wait(tfull(b, blk), ph, abort_flag)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t t0 = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((2 * b + blk) * NMAX);
            uint32_t v[NMAX];
#pragma unroll
            for (int c = 0; c < NMAX; c += 32) if (c < t.n16) tmem_ld32(t0 + c, v + c);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty(b, blk));
            const int j = t.mt * 2 * BLK + blk * BLK + (PAIR ? quad * 16 + (lane & 15) : quad * 32 + lane);
            const bool upper = lane >= 16, b2 = (lane & 4) != 0;
            /* pair: lane and lane ^ 4 hold k = j and j + 4, neighbours in the stored order: the lower one stores both hi, the upper both lo */
            __half *pp = PAIR ? (b2 ? s.out_lo : s.out_hi) + kperm(j & ~4) + (size_t)(t.row0 + (upper ? 1 : 0)) * s.rows : nullptr;
#pragma unroll 1
            for (int c0 = 0; c0 < t.nv; c0 += 32) {
                int rm = t.row0 + c0 + lane;
                if (!PAIR && s.rowmap) rm = c0 + lane < t.nv ? __ldcg(s.rowmap + rm) : 0;
#pragma unroll
                for (int n = 0; n < 32; n += PAIR ? 4 : 2) {
                    if (c0 + n >= t.nv) break;                          /* warp-uniform */
                    if (PAIR) {
                        /* lanes 0-15 hold gate rows, 16-31 the up rows of the same outputs: the lower half finishes columns n and n + 2, the upper n + 1, n + 3 */
                        /* Issue-bound: four columns at a time, so that one exchange carries the hi and lo halves of two of them and the conversions
                         * are packed. 30 layers: 37 tokens 5650 -> 5530 us, 4096 tokens 55.7 -> 54.8 ms, 717 tokens the same. */
                        const uint32_t ga = __shfl_xor_sync(0xffffffffu, upper ? v[n] : v[n + 1], 16), gb = __shfl_xor_sync(0xffffffffu, upper ? v[n + 2] : v[n + 3], 16);
                        const float2 h = make_float2(gelu_mul(__uint_as_float(upper ? ga : v[n]), __uint_as_float(upper ? v[n + 1] : ga)),
                                                     gelu_mul(__uint_as_float(upper ? gb : v[n + 2]), __uint_as_float(upper ? v[n + 3] : gb)));
                        const __half2 x = __floats2half2_rn(h.x, h.y);
                        const float2 xf = __half22float2(x);
                        const __half2 y = __floats2half2_rn(__fsub_rn(h.x, xf.x), __fsub_rn(h.y, xf.y));
                        const uint32_t hx = *reinterpret_cast<const uint32_t *>(&x), hy = *reinterpret_cast<const uint32_t *>(&y);
                        const uint32_t other = __shfl_xor_sync(0xffffffffu, b2 ? hx : hy, 4), a0 = b2 ? other : hx, a1 = b2 ? hy : other;
                        const int nn = c0 + n + (upper ? 1 : 0);
                        if (nn < t.nv) *reinterpret_cast<uint32_t *>(pp) = __byte_perm(a0, a1, 0x5410);
                        if (nn + 2 < t.nv) *reinterpret_cast<uint32_t *>(pp + 2 * (size_t)s.rows) = __byte_perm(a0, a1, 0x7632);
                        pp += 4 * (size_t)s.rows;
                    } else {
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const int r = __shfl_sync(0xffffffffu, rm, n + k);
                            if (c0 + n + k < t.nv && j < s.rows) s.out_f[(size_t)r * s.out_stride + j] = __uint_as_float(v[n + k]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i + 32 < NMAX; i++) v[i] = v[i + 32];
            }
        }
    } else if (warp < kMma) {
        /* ---------------- weights: packed codes in shared memory -> fp16 hi/lo in TMEM; one thread per weight row */
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kUnpRegs));
        const int quad = warp & 3, blk = ((warp - kEpiWarps) >> 2) & 1, set = (warp - kEpiWarps) >> 3;
        const int half = PAIR ? lane >> 4 : 0;
        const int rb = PAIR ? quad * 16 + (lane & 15) : quad * 32 + lane;                /* row inside the block (pair: of its gate or up half) */
        const int box = blk * 2 + (PAIR ? half : rb >> 6), r64 = rb & 63;
        const uint32_t coff = (uint32_t)box * kBoxBytes + (uint32_t)r64 * 128u, r7 = r64 & 7;
        const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + C::kACol + kBK * blk;
        const uint32_t m1032 = in_register(0x64086408u), m72 = in_register(0x54805480u);
        uint32_t as = set, aph = 0, cs = 0, cph = 0;
        int u = set;                                                    /* next stage (64 k) of this set, within the tile; the sets alternate across tiles too */
        /* This thread's block scales travel two chunks (8 scales each) ahead of their use, by asynchronous copies into a
         * place of its own. */
        const uint32_t slot0 = smem_u32(smem) + C::kScaleOff + 16u * (threadIdx.x - 32 * kEpiWarps);
        constexpr uint32_t kSlot = 16u * 32u * C::kUnpWarps;
        int pi = 0, pk = 0, pKB = 0; uint32_t pslot = 0, uslot = 0;     /* next chunk to fetch: item, first 64-k step; slots of a ring of three */
        const uint32_t *sp = nullptr;
        auto fetch = [&]() {
            if (pk == 0 && pKB >= 0) {
                const Item &t = items[pi % kItems];
                pKB = announced(pi) ? t.KB : 0;
                if (pKB == 0) pKB = -1;                                 /* no more */
                else {
                    const TcSeg &s = a.seg[t.sg];
                    int jj = t.mt * 2 * BLK + blk * BLK + rb;
                    if (jj > s.rows - 1) jj = s.rows - 1;
                    const size_t row = (size_t)((long long)t.grp * s.group_rows) + (size_t)(half ? s.up_off : 0) + (size_t)jj;
                    sp = reinterpret_cast<const uint32_t *>(s.bs[half] + row * (size_t)(2 * t.KB));
                }
            }
            if (pKB > 0) {
                const uint32_t dst = slot0 + pslot * kSlot;
                if ((pKB & 3) == 0) asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(sp + pk) : "memory");      /* K a multiple of 256: rows of 16 bytes */
                else {
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (pk + k < pKB) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4u * k), "l"(sp + pk + k) : "memory");
                }
                pk += 4;
                if (pk >= pKB) { pk = 0; pi++; }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            pslot = pslot == 2 ? 0 : pslot + 1;
        };
        fetch(); fetch();
        for (int iw = 0; !failed; iw++) {
            if (!announced(iw)) { failed = true; break; }
            const int KB = items[iw % kItems].KB, nst = blk < items[iw % kItems].nblk ? KB : 0;
            read(iw);
            if (KB == 0) break;
            for (int c0 = 0; c0 < KB; c0 += 4) {
                fetch();
                asm volatile("cp.async.wait_group 2;" ::: "memory");
                const uint32_t sc = slot0 + uslot * kSlot;
                uslot = uslot == 2 ? 0 : uslot + 1;
                if (!mbar_wait(cfull(cs), cph, abort_flag)) { failed = true; break; }
                const unsigned char *codes = smem + C::kCOff + cs * kChunkBytes + coff;
                const int lim = nst < c0 + 4 ? nst : c0 + 4;
#pragma unroll 1                                                        /* one copy of the unpack: several would not stay in the instruction cache */
                for (; u < lim; u += C::kSets) {
                    const int k = u - c0;
                    const uint32_t td = ta + C::kACols * as;
                    uint32_t s2;
                    const int4 w0 = *reinterpret_cast<const int4 *>(codes + (((2 * k) ^ r7) << 4)), w1 = *reinterpret_cast<const int4 *>(codes + (((2 * k + 1) ^ r7) << 4));
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(s2) : "r"(sc + 4u * k));
                    if (!mbar_wait(aempty(as, blk), aph ^ 1, abort_flag)) { failed = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    unpack_block<TERMS >= 3>(w0, (unsigned short)(s2 & 0xFFFFu), m1032, m72, td, td + 32u);
                    unpack_block<TERMS >= 3>(w1, (unsigned short)(s2 >> 16), m1032, m72, td + 16u, td + 48u);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    mbar_arrive_lane0(afull(as, blk), lane);
                    as += C::kSets;
                    if (as >= C::kAStages) { as -= C::kAStages; aph ^= 1; }
                }
                if (failed) break;
                mbar_arrive_lane0(cempty(cs), lane);
                if (++cs == C::kCStages) { cs = 0; cph ^= 1; }
            }
            u -= nst;
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kMiscRegs));
        if (warp < kActs) {
            /* ---------------- MMA issue, a warp per block: the whole warp walks the loop, one lane issues. An MMA of 16 columns
             * keeps the tensor core busy for some ten cycles, and every wait and commit costs about a hundred: the two blocks'
             * chains of them run side by side. */
            const bool leader = elect_one();
            const int blk = warp - kMma;
            uint32_t as = 0, aph = 0, bs = 0, bp = 0; int lt = 0;
            for (int iw = 0; !failed; iw++) {
                if (!announced(iw)) { failed = true; break; }
                const int KB = items[iw % kItems].KB, n16 = items[iw % kItems].n16;
                const bool mine = blk < items[iw % kItems].nblk;
                read(iw);
                if (KB == 0) break;
                const uint32_t idesc = (1u << 4) | ((uint32_t)(n16 >> 3) << 17) | ((128u >> 4) << 24);   /* f16 x f16 -> f32, K-major B, M = 128, N = n16 */
                const int b = lt % C::kAccBufs; const uint32_t bph = (lt / C::kAccBufs) & 1;
                if (mine) {
                    lt++;
                    if (!mbar_wait(tempty(b, blk), bph ^ 1, abort_flag)) { failed = true; break; }
                }
                const uint32_t d = tmem + (uint32_t)((2 * b + blk) * NMAX);
                for (int kb = 0; kb < KB; kb++) {
                    if (mine) {
                        const uint64_t x0 = make_desc(sbase + bs * C::kBStage);
                        /* both at once: a poll takes about a hundred cycles, and a stage some 740 (30 layers of 37 tokens: 5285 -> 5238 us) */
                        if (!mbar_try2(bfull(bs), bp, afull(as, blk), aph) && (!mbar_wait(bfull(bs), bp, abort_flag) || !mbar_wait(afull(as, blk), aph, abort_flag))) { failed = true; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (leader) {
                            const uint32_t wa = tmem + C::kACol + C::kACols * as + kBK * blk;
#pragma unroll
                            for (int ks = 0; ks < kBK / 16; ks++) {
                                const uint64_t xhi = x0 + 2u * ks, xlo = xhi + 8u * (uint32_t)n16;       /* 32 bytes along k; the lo rows behind the hi rows */
                                if (ks == 0) umma_f16_ts(d, wa, xhi, idesc, kb ? 1u : 0u); else umma_f16_ts(d, wa + 8u * ks, xhi, idesc);
                                if (TERMS >= 3) umma_f16_ts(d, wa + kBK / 2 + 8u * ks, xhi, idesc | kNegateA);
                                if (TERMS >= 2) umma_f16_ts(d, wa + 8u * ks, xlo, idesc);
                            }
                            umma_commit(aempty(as, blk));               /* both stages are free once these MMAs have read them */
                            umma_commit(bempty(bs));
                            if (kb + 1 == KB) umma_commit(tfull(b, blk));
                        }
                        __syncwarp();
                        if (++as == C::kAStages) { as = 0; aph ^= 1; }
                    } else {
                        if (!mbar_wait(bfull(bs), bp, abort_flag)) { failed = true; break; }
                        mbar_arrive_lane0(bempty(bs), lane);
                    }
                    if (++bs == C::kBStages) { bs = 0; bp ^= 1; }
                }
            }
        } else if (warp == kActs) {
            /* ---------------- activation rows by TMA. (Four gathered rows a copy, tile::gather4 from one
             * row per token, would save the sorted copy of the rows, but such copies are too slow: 1640 against 870 us for the
             * gate|up launch of 4096 tokens.) */
            if (lane == 0) {                                            /* one lane walks the loop: with the warp in step this chain paces the CTA (30 layers of 24 tokens: +7%) */
                uint32_t bs = 0, bp = 0;
                for (int iw = 0; !failed; iw++) {
                    if (!announced(iw)) { failed = true; break; }
                    const int KB = items[iw % kItems].KB, n16 = items[iw % kItems].n16, sg = items[iw % kItems].sg, row0 = items[iw % kItems].row0;
                    mbar_arrive(iempty(iw));
                    if (KB == 0) break;
                    /* hi and lo rows of a whole tile in one copy, a map per height: this lane's chain of wait, expect and copies is what
                     * paces the CTA. In copies of 16 or 64 rows of hi or lo (6 for a tile of 48), 30 layers of 400 / 717 / 1500 tokens took
                     * 9.38 / 12.6 / 23.2 ms instead of 9.15 / 12.1 / 22.6; of 37 tokens (2 copies) the same. */
                    const CUtensorMap *map = &maps.act[sg][n16 / kNGran - 1];
                    for (int kb = 0; kb < KB; kb++) {
                        if (!mbar_wait(bempty(bs), bp ^ 1, abort_flag)) { failed = true; break; }
                        const uint32_t dst = sbase + bs * C::kBStage, bar = bfull(bs);
                        mbar_expect_tx(bar, (uint32_t)n16 * (TERMS >= 2 ? 256u : 128u));
                        tma_load_3d(dst, map, kb * kBK, row0, 0, bar);
                        if (++bs == C::kBStages) { bs = 0; bp ^= 1; }
                    }
                }
            }
            if (failed || *abort_flag) __nanosleep(100000);             /* let copies in flight land before the CTA leaves */
        } else if (warp == kCodes && lane == 0) {
            /* ---------------- the tiles, and their packed codes by TMA, 256 k a copy. A CTA's first tile is its own number; each
             * next one is drawn from a counter when the codes of the one before are on their way, some 16 stages before it is due.
             * Tiles differ: the shared expert's K is three times the routed experts' in the down GEMM, the last tile of a group's
             * rows may hold one block, and a CTA draws four to ten tiles in all when there are few rows. Dealt out in turn
             * (CTA c: c, c + 148, ...), the CTAs with a long tile got as many others as the rest: a layer of 24 / 37 / 400 / 717 tokens takes
             * 165 / 180 / 299 / 392 us so, 148 / 168 / 293 / 386 drawn, all else the same. The order stays: shared expert first,
             * so the long tiles are out early. */
            const int total0 = *a.seg[0].n_tiles * a.seg[0].m_tiles;
            const int total = total0 + (a.nseg > 1 ? *a.seg[1].n_tiles * a.seg[1].m_tiles : 0);
            uint32_t cc = 0;
            for (int w = blockIdx.x, i = 0; !failed; w = (int)gridDim.x + atomicAdd(a.ticket, 1), i++) {
                if (!mbar_wait(iempty(i), ((uint32_t)(i / kItems) & 1u) ^ 1u, abort_flag)) { failed = true; break; }
                /* work item -> segment, activation tile, weight tile (the weight tiles of one activation tile are neighbours) */
                Item t;
                t.sg = w >= total0 ? 1 : 0;
                const TcSeg &s = a.seg[t.sg];
                t.KB = 0;
                if (w < total) {
                    const int r = w - (t.sg ? total0 : 0), nt = r / s.m_tiles;
                    t.mt = r - nt * s.m_tiles;
                    t.grp = __ldcg(s.tiles + 3 * nt); t.row0 = __ldcg(s.tiles + 3 * nt + 1); t.nv = __ldcg(s.tiles + 3 * nt + 2);
                    t.n16 = (t.nv + kNGran - 1) & ~(kNGran - 1);
                    t.nblk = s.rows - t.mt * 2 * BLK > BLK ? 2 : 1;
                    t.KB = a.K[t.sg] / kBK;
                }
                items[i % kItems] = t;
                mbar_arrive(ifull(i));
                if (t.KB == 0) break;
                const int y0 = (int)((long long)t.grp * s.group_rows) + t.mt * 2 * BLK;
                for (int kc = 0; kc < t.KB; kc += 4, cc++) {
                    const uint32_t cs = cc % C::kCStages, cp = (cc / C::kCStages) & 1;
                    if (!mbar_wait(cempty(cs), cp ^ 1, abort_flag)) { failed = true; break; }
                    mbar_expect_tx(cfull(cs), 2u * t.nblk * kBoxBytes);
                    const uint32_t dst = sbase + C::kCOff + cs * kChunkBytes;
                    for (int q = 0; q < 2 * t.nblk; q++) {
                        const int y = y0 + (q >> 1) * BLK + (PAIR ? (q & 1 ? s.up_off : 0) : 64 * (q & 1));
                        tma_load_2d(dst + kBoxBytes * q, &maps.codes[t.sg][PAIR ? q & 1 : 0], kc * 32, y, cfull(cs));
                    }
                }
            }
            if (failed || *abort_flag) __nanosleep(100000);
        }
        __syncwarp();
    }
    if (failed && lane == 0) atomicExch(a.status, SP_KERR_BARRIER_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kCodes) {
        if (*abort_flag) __nanosleep(100000);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

/* ---------------------------------------------------------------- helpers around the GEMM */
/* fp32 rows -> fp16 hi/lo rows, k order 0,4,1,5,2,6,3,7 inside each group of 8; one block per row */
__global__ void __launch_bounds__(256) k_tc_split(const float *src, const int *gather, int K, __half *hi, __half *lo) {
    const size_t r = blockIdx.x;
    const float *x = src + (size_t)(gather ? gather[r] : (int)r) * K;
    for (int c = threadIdx.x; c < K / 8; c += 256) {
        const float4 a = *reinterpret_cast<const float4 *>(x + 8 * c), b = *reinterpret_cast<const float4 *>(x + 8 * c + 4);
        const float v[8] = {a.x, b.x, a.y, b.y, a.z, b.z, a.w, b.w};
        __half h[8], l[8];
#pragma unroll
        for (int k = 0; k < 8; k++) { h[k] = __float2half_rn(v[k]); l[k] = __float2half_rn(__fsub_rn(v[k], __half2float(h[k]))); }
        *reinterpret_cast<uint4 *>(hi + r * K + 8 * c) = *reinterpret_cast<const uint4 *>(h);
        *reinterpret_cast<uint4 *>(lo + r * K + 8 * c) = *reinterpret_cast<const uint4 *>(l);
    }
}
/* fp16 hi/lo rows of the tokens -> the rows of the pairs, sorted by expert; one block per sorted row, one thread per 16 bytes
 * of hi and of lo */
__global__ void __launch_bounds__(512) k_tc_permute(const __half *src_hi, const __half *src_lo, const int *gather, int K, __half *hi, __half *lo) {
    sp_pdl_wait();
    sp_pdl_next();
    const size_t r = (size_t)blockIdx.x * (K / 8), s = (size_t)gather[blockIdx.x] * (K / 8);
    const int c = threadIdx.x;
    if (c >= K / 8) return;
    const uint4 h = reinterpret_cast<const uint4 *>(src_hi)[s + c], l = reinterpret_cast<const uint4 *>(src_lo)[s + c];
    reinterpret_cast<uint4 *>(hi)[r + c] = h; reinterpret_cast<uint4 *>(lo)[r + c] = l;
}
/* block-wide inclusive scan of one int per thread (1024 threads) */
__device__ __forceinline__ int scan1024(int v, int *sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
    if (lane == 31) sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int t = sh[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, t, o); if (lane >= o) t += u; }
        sh[lane] = t;
    }
    __syncthreads();
    const int r = v + (warp ? sh[warp - 1] : 0);
    __syncthreads();
    return r;
}
/* activation tiles: each group's rows in the fewest tiles of at most nmax rows, evenly sized (a multiple of 16). One
 * thread per group (groups <= 1024) counts its tiles, a scan places them, each thread writes its own. Row ranges are
 * clamped to [0, max_rows]: offsets come from the caller (or from counts another GPU sent). Block-wide. */
__device__ __forceinline__ void write_tiles(int first, int cnt, int nmax, int *tiles, int *n_tiles, int cap, int *sh) {
    const int nt = cnt > 0 ? (cnt + nmax - 1) / nmax : 0;
    const int per = nt > 0 ? ((((cnt + nt - 1) / nt) + kNGran - 1) & ~(kNGran - 1)) : 0;
    const int mine = nt > 0 ? (cnt + per - 1) / per : 0;
    const int end = scan1024(mine, sh);
    int n = end - mine;
    for (int i = 0; i < mine && n < cap; i++, n++) {
        const int left = cnt - i * per;
        tiles[3 * n] = (int)threadIdx.x; tiles[3 * n + 1] = first + i * per; tiles[3 * n + 2] = left < per ? left : per;
    }
    if (threadIdx.x == 1023) { *n_tiles = end < cap ? end : cap; n_tiles[1] = n_tiles[2] = 0; }
}
__global__ void __launch_bounds__(1024) k_tc_plan(const int *offsets, int groups, int fixed_rows, int max_rows, int nmax, int *tiles, int *n_tiles, int cap) {
    __shared__ int sh[32];
    const int g = threadIdx.x;
    int first = 0, cnt = 0;
    if (g < groups) {
        first = offsets ? offsets[g] : 0;
        int last = offsets ? offsets[g + 1] : fixed_rows;
        first = first < 0 ? 0 : (first > max_rows ? max_rows : first);
        last = last < first ? first : (last > max_rows ? max_rows : last);
        cnt = last - first;
    }
    write_tiles(first, cnt, nmax, tiles, n_tiles, cap, sh);
}
/* one launch between the router and the GEMMs: every block scans the per-expert counts for itself and places 1024
 * pairs (sorted row = the expert's first row + the pair's position in its list); block 0 also writes the tile tables
 * of the routed rows and of the M rows of the shared expert */
struct SortArgs {
    const int *count, *sel_asc, *pairpos; int groups, M, NU, nmax;
    int *gather, *rowmap, *tiles_r, *n_r, *tiles_sh, *n_sh; int cap_r, cap_sh;
};
__global__ void __launch_bounds__(1024) k_tc_sort(SortArgs s) {
    __shared__ int sh[32];
    __shared__ int off[1024];
    sp_pdl_wait();
    sp_pdl_next();
    const int t = threadIdx.x, cnt = t < s.groups ? s.count[t] : 0;
    const int first = scan1024(cnt, sh) - cnt;
    off[t] = first;
    __syncthreads();
    const int p = blockIdx.x * 1024 + t;
    if (p < s.M * s.NU) {
        const int row = off[s.sel_asc[p]] + s.pairpos[p];
        s.gather[row] = p / s.NU; s.rowmap[row] = p;
    }
    if (blockIdx.x == 0) {
        write_tiles(first, cnt, s.nmax, s.tiles_r, s.n_r, s.cap_r, sh);
        write_tiles(0, t == 0 ? s.M : 0, s.nmax, s.tiles_sh, s.n_sh, s.cap_sh, sh);
    }
}

}  // namespace

/* ---------------------------------------------------------------- host side */
struct SpTcPlan {
    int Mcap, Rcap, sms;
    unsigned char *base; size_t bytes;
    __half *nx_hi, *nx_lo, *hd_hi, *hd_lo, *in_hi, *in_lo, *h_hi, *h_lo, *tk_hi, *tk_lo;           /* tk: the routed experts' input, one row per token; in: one per pair */
    int *tiles_sh, *ntiles_sh, *tiles_r, *ntiles_r, *gather, *rowmap;
    int cap_sh, cap_r;
    int terms;                                         /* MMAs per k-step: 3, 2 or 1 */
    CUtensorMap nx[4], hd[4], in[4], h[4];             /* boxes of 16, 32, 48 and 64 rows, hi and lo */
    sp_tc::EncodeTiledFn encode;
    std::map<const void *, CUtensorMap> codes;         /* one per weight tensor of the arena, made at first use */
};

void sp_tc_inputs(SpTcPlan *p, __half **nx_hi, __half **nx_lo, __half **in_hi, __half **in_lo) { *nx_hi = p->nx_hi; *nx_lo = p->nx_lo; *in_hi = p->tk_hi; *in_lo = p->tk_lo; }
bool sp_tc_supported(const SpDims &d) { return (d.E % 64 == 0) && (d.FFE % 64 == 0) && (d.FFS % 64 == 0); }

namespace {
/* [plane][row][element], boxes of box_planes x box_rows rows of 128 bytes */
cudaError_t make_map(sp_tc::EncodeTiledFn fn, CUtensorMap *m, CUtensorMapDataType type, const void *ptr, size_t row_elems, size_t row_bytes, size_t rows, int planes, int box_elems, int box_rows, int box_planes) {
    const cuuint64_t dims[3] = {(cuuint64_t)row_elems, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)(row_bytes * rows)};
    const cuuint32_t box[3] = {(cuuint32_t)box_elems, (cuuint32_t)box_rows, (cuuint32_t)box_planes};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(m, type, planes > 1 ? 3 : 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
/* the packed codes of one weight tensor: rows of K/2 bytes, boxes of 128 bytes x 64 rows (what lies past either edge reads as zero) */
cudaError_t codes_map(SpTcPlan *p, const uint8_t *codes, int K, size_t rows, CUtensorMap *out) {
    auto it = p->codes.find(codes);
    if (it == p->codes.end()) {
        CUtensorMap m;
        const cudaError_t e = make_map(p->encode, &m, CU_TENSOR_MAP_DATA_TYPE_UINT8, codes, (size_t)K / 2, (size_t)K / 2, rows, 1, 128, (int)kBoxRows, 1);
        if (e != cudaSuccess) return e;
        it = p->codes.emplace(codes, m).first;
    }
    *out = it->second;
    return cudaSuccess;
}
size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

template <bool PAIR, int TERMS, int NMAX>
cudaError_t prepare_kernel() {
    cudaFuncAttributes at;
    cudaError_t e = cudaFuncGetAttributes(&at, k_tc_gemm<PAIR, TERMS, NMAX>);
    if (e != cudaSuccess) return e;
    if (at.numRegs != Cfg<NMAX>::kLaunchRegs) return cudaErrorInvalidConfiguration;      /* the register split counts on it */
    return cudaFuncSetAttribute(k_tc_gemm<PAIR, TERMS, NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<NMAX>::kSmem);
}
template <int TERMS>
cudaError_t prepare_terms() {
    cudaError_t e = prepare_kernel<true, TERMS, 32>();
    if (e == cudaSuccess) e = prepare_kernel<false, TERMS, 32>();
    if (e == cudaSuccess) e = prepare_kernel<true, TERMS, 64>();
    if (e == cudaSuccess) e = prepare_kernel<false, TERMS, 64>();
    return e;
}
}  // namespace

cudaError_t sp_tc_create(const SpDims &d, int max_tokens, int max_rows, SpTcPlan **out, size_t *bytes) {
    *out = nullptr; *bytes = 0;
    if (!sp_tc_supported(d)) return cudaSuccess;
    sp_tc::EncodeTiledFn fn = nullptr;
    cudaError_t e = sp_tc::encode_tiled_fn(&fn);
    if (e != cudaSuccess) return e;
    SpTcPlan *p = new SpTcPlan();
    p->encode = fn;
    p->Mcap = ((max_tokens + 127) / 128) * 128;
    p->Rcap = (int)((((long long)max_rows + 127) / 128) * 128);
    int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, dev);
    p->cap_sh = p->Mcap / 32 + 2; p->cap_r = p->Rcap / 32 + d.NE + 2;
    size_t o = 0; auto take = [&](size_t b) { size_t at = o; o = up256(o + b); return at; };
    const size_t E = d.E, FFE = d.FFE, FFS = d.FFS, Mc = p->Mcap, Rc = p->Rcap;
    const size_t o_nx = take(4 * Mc * E), o_hd = take(4 * Mc * FFS), o_in = take(4 * Rc * E), o_h = take(4 * Rc * FFE), o_tk = take(4 * Mc * E);      /* hi rows, then lo rows */
    const size_t o_tsh = take(12 * (size_t)p->cap_sh), o_nsh = take(12), o_tr = take(12 * (size_t)p->cap_r), o_nr = take(12);
    const size_t o_g = take(4 * Rc), o_rm = take(4 * Rc);
    p->bytes = o;
    e = cudaMalloc((void **)&p->base, o);
    if (e != cudaSuccess) { delete p; return e; }
    cudaMemset(p->base, 0, o);
    unsigned char *b = p->base;
    p->nx_hi = (__half *)(b + o_nx); p->nx_lo = p->nx_hi + Mc * E; p->hd_hi = (__half *)(b + o_hd); p->hd_lo = p->hd_hi + Mc * FFS;
    p->in_hi = (__half *)(b + o_in); p->in_lo = p->in_hi + Rc * E; p->h_hi = (__half *)(b + o_h); p->h_lo = p->h_hi + Rc * FFE;
    p->tk_hi = (__half *)(b + o_tk); p->tk_lo = p->tk_hi + Mc * E;
    p->tiles_sh = (int *)(b + o_tsh); p->ntiles_sh = (int *)(b + o_nsh); p->tiles_r = (int *)(b + o_tr); p->ntiles_r = (int *)(b + o_nr);
    p->gather = (int *)(b + o_g); p->rowmap = (int *)(b + o_rm);
    /* house convention: behaviour switches are SP_* variables read once. 3 (default) keeps every product the fp32
     * reference arithmetic sees down to 2^-22; 2 rounds the dequantised weight to fp16; 1 also rounds the activation. */
    const char *tv = getenv("SP_MOE_PREFILL_TERMS");
    p->terms = tv ? atoi(tv) : 3;
    if (p->terms < 1 || p->terms > 3) p->terms = 3;
    cudaError_t m = cudaSuccess;
    auto mk = [&](CUtensorMap *t, const __half *hi, size_t K, size_t rows) {
        for (int i = 0; i < kNMax / kNGran && m == cudaSuccess; i++)
            m = make_map(fn, t + i, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, hi, K, 2 * K, rows, 2, kBK, (i + 1) * kNGran, p->terms >= 2 ? 2 : 1);
    };
    mk(p->nx, p->nx_hi, E, Mc); mk(p->hd, p->hd_hi, FFS, Mc);
    mk(p->in, p->in_hi, E, Rc); mk(p->h, p->h_hi, FFE, Rc);
    if (m == cudaSuccess) m = p->terms == 3 ? prepare_terms<3>() : p->terms == 2 ? prepare_terms<2>() : prepare_terms<1>();
    if (m != cudaSuccess) { cudaFree(p->base); delete p; return m; }
    *out = p; *bytes = o;
    return cudaSuccess;
}
void sp_tc_destroy(SpTcPlan *p) { if (!p) return; if (p->base) cudaFree(p->base); delete p; }

namespace {
/* activation rows per tile: tiles of 32 have a second set of accumulators, tiles of 64 serve more rows per unpacked weight. The
 * line is at 12 rows per expert, and at 16 where tiles of 64 would be fewer than the SMs. Us a layer with 32 / 64, E 2816, 128 experts,
 * 8 each, FFE 704: 146 / 153 at 24 tokens, 189 / 193 at 64, 208 / 214 at 130 (8 rows per expert), 210 / 215 at 160, 219 / 223 at 200,
 * 255 / 256 at 256, 312 / 298 at 400. With a router that sends most tokens to a few experts (Zipf 1.2) 129 / 117 at 130,
 * 148 / 127 at 200, 171 / 139 at 256: what a line above 12 gives the even one it takes several times from that one. With 64 experts, 6
 * each, E 2048, FFE 1408: 153 / 159 at 100 (9 rows), 156 / 162 at 130, 173 / 172 at 170 (16 rows), Zipf 130 / 112. With 32, 4 each, E
 * 1024, FFE 512, 136 tiles of gate|up with 64: 42 / 50 at 64 (8 rows), 47 / 56 at 128, 62.8 / 61.7 at 200 (25 rows). groups: the experts that the
 * rows can belong to; M: rows of the shared expert in the same launch. */
int tile_rows(const SpTcPlan *p, const SpDims &d, int groups, long long rows, int M) {
    const long long tiles = (long long)groups * ((d.FFE + 127) / 128) + (long long)((M + 63) / 64) * ((d.FFS + 127) / 128);
    return rows > (tiles < p->sms ? 16LL : 12LL) * groups ? 64 : 32;
}

template <bool PAIR, int NMAX>
cudaError_t launch_n(const SpTcPlan *p, const TcArgs &a, const TcMaps &maps, cudaStream_t st, int *nl) {
    return sp_launch(p->terms == 3 ? k_tc_gemm<PAIR, 3, NMAX> : p->terms == 2 ? k_tc_gemm<PAIR, 2, NMAX> : k_tc_gemm<PAIR, 1, NMAX>,
                     dim3((unsigned)p->sms), Cfg<NMAX>::kThreads, Cfg<NMAX>::kSmem, st, nl, a, maps);
}
/* the GEMMs of one launch, at most two (the shared expert's and the routed experts') */
struct Launch {
    SpTcPlan *p; const SpDims &d; const SpLayerDev &L; TcArgs a{}; TcMaps maps; cudaError_t err = cudaSuccess;
    Launch(SpTcPlan *p_, const SpDims &d_, const SpLayerDev &L_, int *status) : p(p_), d(d_), L(L_) { a.status = status; }
    TcSeg &seg(int K, const CUtensorMap *act, const uint8_t *c0, const uint16_t *b0, const uint8_t *c1, const uint16_t *b1, size_t tensor_rows, int rows, int m_tiles) {
        const int i = a.nseg++;
        a.K[i] = K;
        for (int n = 0; n < kNMax / kNGran; n++) maps.act[i][n] = act[n];
        if (err == cudaSuccess) err = codes_map(p, c0, K, tensor_rows, &maps.codes[i][0]);
        if (err == cudaSuccess) err = codes_map(p, c1, K, tensor_rows, &maps.codes[i][1]);
        TcSeg &s = a.seg[i];
        s.bs[0] = b0; s.bs[1] = b1; s.rows = rows; s.m_tiles = m_tiles;
        return s;
    }
    void shared_up() {
        TcSeg &s = seg(d.E, p->nx, L.sg_codes, L.sg_bs, L.su_codes, L.su_bs, d.FFS, d.FFS, (d.FFS + 127) / 128);
        s.tiles = p->tiles_sh; s.n_tiles = p->ntiles_sh; s.out_hi = p->hd_hi; s.out_lo = p->hd_lo;
    }
    void shared_down(float *dn) {
        TcSeg &s = seg(d.FFS, p->hd, L.sd_codes, L.sd_bs, L.sd_codes, L.sd_bs, d.E, d.E, (d.E + 255) / 256);
        s.tiles = p->tiles_sh; s.n_tiles = p->ntiles_sh; s.out_f = dn; s.out_stride = d.E;
    }
    void routed_up() {
        TcSeg &s = seg(d.E, p->in, L.gu_codes, L.gu_bs, L.gu_codes, L.gu_bs, (size_t)d.NE * 2 * d.FFE, d.FFE, (d.FFE + 127) / 128);
        s.group_rows = 2LL * d.FFE; s.up_off = d.FFE; s.tiles = p->tiles_r; s.n_tiles = p->ntiles_r; s.out_hi = p->h_hi; s.out_lo = p->h_lo;
    }
    void routed_down(float *out, const int *rowmap) {
        TcSeg &s = seg(d.FFE, p->h, L.dn_codes, L.dn_bs, L.dn_codes, L.dn_bs, (size_t)d.NE * d.E, d.E, (d.E + 255) / 256);
        s.group_rows = d.E; s.tiles = p->tiles_r; s.n_tiles = p->ntiles_r; s.out_f = out; s.out_stride = d.E; s.rowmap = rowmap;
    }
    cudaError_t go(bool pair, int nmax, int *n_tiles, cudaStream_t st, int *nl) {      /* n_tiles: behind the count, the tickets of gate|up and of down */
        a.ticket = n_tiles + (pair ? 1 : 2);
        if (err != cudaSuccess) return err;
        for (int i = a.nseg; i < 2; i++) {
            for (int n = 0; n < kNMax / kNGran; n++) maps.act[i][n] = maps.act[0][n];
            maps.codes[i][0] = maps.codes[i][1] = maps.codes[0][0]; a.K[i] = a.K[0];
        }
        if (pair) return nmax == 64 ? launch_n<true, 64>(p, a, maps, st, nl) : launch_n<true, 32>(p, a, maps, st, nl);
        return nmax == 64 ? launch_n<false, 64>(p, a, maps, st, nl) : launch_n<false, 32>(p, a, maps, st, nl);
    }
};
}  // namespace

cudaError_t sp_tc_layer(SpTcPlan *p, const SpDims &d, const SpLayerDev &L, int M, const int *sel_asc, const int *count, const int *pairpos, float *dn, float *eo,
                        int *status, cudaStream_t st, int *nl) {
    const int R = M * d.NU;
    if (!p || M > p->Mcap || (long long)M * d.NU > p->Rcap) return cudaErrorInvalidValue;
    const int nmax = tile_rows(p, d, d.NE, R, M);
    SortArgs s{count, sel_asc, pairpos, d.NE, M, d.NU, nmax, p->gather, p->rowmap, p->tiles_r, p->ntiles_r, p->tiles_sh, p->ntiles_sh, p->cap_r, p->cap_sh};
    cudaError_t e = sp_launch(k_tc_sort, dim3((unsigned)((R + 1023) / 1024)), 1024, 0, st, nl, s);
    if (e != cudaSuccess) return e;
    e = sp_launch(k_tc_permute, dim3((unsigned)R), (unsigned)((d.E / 8 + 31) & ~31), 0, st, nl, p->tk_hi, p->tk_lo, p->gather, d.E, p->in_hi, p->in_lo);
    if (e != cudaSuccess) return e;
    Launch up(p, d, L, status);
    up.shared_up(); up.routed_up();
    e = up.go(true, nmax, p->ntiles_r, st, nl);
    if (e != cudaSuccess) return e;
    Launch down(p, d, L, status);
    down.shared_down(dn); down.routed_down(eo, p->rowmap);
    return down.go(false, nmax, p->ntiles_r, st, nl);
}

cudaError_t sp_tc_shared_expert(SpTcPlan *p, const SpDims &d, const SpLayerDev &L, int M, const float *nx, float *dn,
                                int *status, cudaStream_t st, int *nl, int phase) {
    if (!p || M > p->Mcap) return cudaErrorInvalidValue;
    const int nmax = M > 32 ? 64 : 32;
    cudaError_t e = cudaSuccess;
    if (phase != 2) {                                     /* gate/up + GeGLU -> hd (split fp16), kept in the plan's scratch */
        k_tc_split<<<M, 256, 0, st>>>(nx, nullptr, d.E, p->nx_hi, p->nx_lo); (*nl)++;
        k_tc_plan<<<1, 1024, 0, st>>>(nullptr, 1, M, M, nmax, p->tiles_sh, p->ntiles_sh, p->cap_sh); (*nl)++;
        Launch up(p, d, L, status);
        up.shared_up();
        e = up.go(true, nmax, p->ntiles_sh, st, nl);
    }
    if (phase != 1 && e == cudaSuccess) {                 /* down: hd -> dn (the tile table of the first phase is still in place) */
        Launch down(p, d, L, status);
        down.shared_down(dn);
        e = down.go(false, nmax, p->ntiles_sh, st, nl);
    }
    return e;
}

cudaError_t sp_tc_routed(SpTcPlan *p, const SpDims &d, const SpLayerDev &L, int R, int owners, const float *src, const int *gather,
                         const int *offsets, const int *rowmap, float *out, int *status, cudaStream_t st, int *nl) {
    if (!p || R > p->Rcap) return cudaErrorInvalidValue;
    if (R == 0) return cudaSuccess;
    /* where the caller does not know how many of the experts are its rank's, the line is at 8 rows per expert of the model: two thirds
     * of it, as they are fewer */
    const int nmax = owners ? tile_rows(p, d, owners, R, 0) : tile_rows(p, d, d.NE, 3LL * R / 2, 0);
    k_tc_split<<<R, 256, 0, st>>>(src, gather, d.E, p->in_hi, p->in_lo); (*nl)++;
    k_tc_plan<<<1, 1024, 0, st>>>(offsets, d.NE, 0, R, nmax, p->tiles_r, p->ntiles_r, p->cap_r); (*nl)++;
    Launch up(p, d, L, status);
    up.routed_up();
    cudaError_t e = up.go(true, nmax, p->ntiles_r, st, nl);
    if (e != cudaSuccess) return e;
    Launch down(p, d, L, status);
    down.routed_down(out, rowmap);
    return down.go(false, nmax, p->ntiles_r, st, nl);
}
