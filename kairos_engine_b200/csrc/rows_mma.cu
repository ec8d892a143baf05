/* rows_mma.cu — Q4B rows x the int8 activations of a list of tokens, in the decode arithmetic, for M > 1.
 *
 * The sums are those of k_gemv_q4b_dp4a_v2 (CF:1688-1713 of src/backends/cuda/cuda_forward.cu), bit for bit: for every
 * (row, token) the 32-weight chunk c adds fma(scale, fma(a0, s0, a1 * s1), acc) to slot c % 32, chunks in ascending order
 * (a0, a1: exact integer dots of the chunk's two 16-blocks), and the 32 slots are added in the pairing of the shuffle-down
 * tree. What is free is who does it when:
 *   - One mma.sync m16n8k32 (s8 x s8) takes 16 weight rows x one chunk x four tokens: column 2t + h of B is token t
 *     restricted to half h, so lane (g, q) of the warp finds both block sums of rows g and g + 8 for token q in its C
 *     registers, for every chunk. It adds its slots by itself, in the order that completes subtrees (no shuffles, at most
 *     four partial sums waiting). Half of the MMA multiplies zeros; the MMA pipe has room for that (8 cycles per
 *     instruction and scheduler, 16% of the time), and the epilogue's 10 fp32 instructions serve four tokens at a time. While most experts
 *     have one or two tokens, two neighbouring chunks x two tokens share an epilogue instead (W = 2 below).
 *   - A operand: code nibbles moved to the top of a byte (16 * code as s8); C starts at 0x4B400000, so that one fma turns
 *     the s32 result into the float a conversion would give.
 *   - Gate|up: a 16-row MMA tile is 8 gate rows and the 8 up rows of the same outputs. A unit is 16 outputs = one
 *     quantisation block: it leaves the kernel as int8 codes and a scale, ready for the down rows.
 *
 * Work is cut into units of ~50 KB of weights x up to 4 or 16 tokens. One CTA per SM; one warp asks the copy engine for the
 * units' rows (a ring of stages), two teams of eight warps consume them alternately, and a warp per team has the activations
 * of its next four tokens copied while it multiplies the current four. So the weight stream does not stop between units, and experts
 * nobody chose cost nothing. A unit's codes are one or two tensor copies (a box of all 128-byte slices of 16 to 128 rows, swizzled, so that the eight
 * rows an MMA operand takes lie on different banks): a copy costs its warp ~85 cycles whatever its size, and a copy per row (for
 * padded rows) took longer than the multiplication. The multiplying warps bound it: at 16 tokens the launches take 50 + 36 us
 * with units of 16, 46 + 33 without their copies and 31 + 21 without their dots. A team spends some 2200 cycles on a unit's dots
 * (16 warps issue in 75% of them), 900 until the last of its sums is finished by two of them, and 300 to 1000 waiting. One team of
 * sixteen warps on a unit was slower (199 us a layer at 64 tokens against 176), and so were sums finished by a warp of their
 * own (one per team 165, for 160: ~300 instructions a unit are too long a chain for one warp) and four chunks x one token per
 * MMA group (103 at 16 tokens: as many instructions a token).
 */
#include "rows_mma.cuh"
#include "launch.cuh"
#include "tc_common.cuh"
#include <cstring>

namespace {
using namespace sp_tc;

constexpr int kTeamWarps = 8, kTeamThreads = 32 * kTeamWarps, kTok = 4, kMaxStages = 4, kMaxTeams = 2;
constexpr int kFewItems = 24, kManyItems = 48;     /* items to a group up to which units are of 4 tokens: on average, and in any one group */
constexpr int kSmUnits = 16;                       /* ... in one group: where units of 16 are at least this many to an SM */
constexpr int kUnits = 128;                        /* unit descriptors of a CTA kept in shared memory */
constexpr int kMagic = 0x4B400000;

struct SegGeo {                                    /* what the copies and the dots need of a segment's shape */
    int tiles, mt_n, n32;                          /* weight tiles per group, 16-row MMA tiles of one, chunks of a row */
    unsigned sb, box_bytes, scale_off;             /* bytes of a row's scales, of one box of codes; where the scales start in a stage */
    unsigned ast;                                  /* bytes between tokens in a buffer */
};
struct RowsArgs {
    SpRowsSeg seg[2]; SegGeo geo[2]; int nseg;
    int stages, teams;
    int many[2];                                   /* a group of more items than this has units of up to 16 tokens, others of up to 4 */
    unsigned stage_bytes, act_bytes, zero_bytes;   /* one stage; one buffer of four tokens; the zeros B's other columns read */
    int *status;
    CUtensorMap codes[2][2];                       /* [segment][gate or only / up] */
};

/* shapes in shared memory */
unsigned up1024(unsigned v) { return (v + 1023u) & ~1023u; }
int box_rows(const SegGeo &g, bool pair) { return pair ? 16 : 16 * g.mt_n; }
SegGeo seg_geo(const SpRowsSeg &s, bool pair) {
    SegGeo g;
    g.mt_n = pair ? 2 : (s.in <= 1024 ? 8 : 2);
    const int per = box_rows(g, pair);                      /* output rows of a unit */
    g.tiles = (s.rows + per - 1) / per; g.n32 = s.in / 32; g.sb = s.in / 16;
    g.box_bytes = 128u * per * ((s.in / 2 + 127) / 128);
    g.scale_off = (pair ? 2 : 1) * g.box_bytes;
    g.ast = (unsigned)sp_act_pitch(s.in); g.ast += (32 - g.ast % 128 + 128) % 128;         /* = 32 mod 128: four tokens on four bank groups */
    return g;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, unsigned bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
/* a box of codes: all 128-byte slices of some consecutive rows, slice-major, 128-byte swizzle */
__device__ __forceinline__ void box_g2s(uint32_t dst, const CUtensorMap *map, int row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%4, %2, %4}], [%3];" ::"r"(dst), "l"(map), "r"(row), "r"(bar), "r"(0) : "memory");
}

/* D = A x B + {magic, ...}, D += A x B (pure functions of their operands: the compiler may move them) */
__device__ __forceinline__ void mma_s8(int (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1, int c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void mma_s8_add(int (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
/* bits of magic + 16 S -> float(S), for two neighbouring registers at once (a layer of 64 tokens 162.6 -> 159.0 us, of 16 86.7 -> 86.1) */
__device__ __forceinline__ float2 magic_to_float2(int a, int b) {
    float2 r;
    asm("{ .reg .b64 v, m, c; mov.b64 v, {%2, %3}; mov.b64 m, {%4, %4}; mov.b64 c, {%5, %5}; fma.rn.f32x2 v, v, m, c; mov.b64 {%0, %1}, v; }"
        : "=f"(r.x), "=f"(r.y) : "r"(a), "r"(b), "f"(0.0625f), "f"(-786432.0f));
    return r;
}

/* ---------------------------------------------------------------- units of work */
struct Unit { int seg, grp, tile, t0, nt; };                /* weight tile `tile` of group grp x its tokens [t0, t0 + nt) */
struct UnitWord { unsigned w; int t0; };                    /* the same as it is kept: nt 5 bits, seg 1, grp 10, tile 16 */
__device__ __forceinline__ UnitWord pack(const Unit &u) { return UnitWord{(unsigned)u.nt | (unsigned)u.seg << 5 | (unsigned)u.grp << 6 | (unsigned)u.tile << 16, u.t0}; }
__device__ __forceinline__ Unit unpack(const UnitWord &p) { return Unit{(int)(p.w >> 5 & 1u), (int)(p.w >> 6 & 1023u), (int)(p.w >> 16), p.t0, (int)(p.w & 31u)}; }
struct Plan {                                               /* in shared memory: first unit of every group, per segment */
    const int *start[2]; int total[2];
    const int *count;                                       /* items of segment 1's groups while the table is in place, else NULL */
};
/* counts, lists and ranges are written by the kernel before this one, which may still run when this one starts: no read-only
 * (__ldg) loads, which the compiler may move before the wait for it */
__device__ __forceinline__ int group_first(const SpRowsSeg &s, int g) {
    if (!s.offset) return 0;
    const int f = __ldcg(s.offset + g);                      /* caller-supplied ranges: kept inside the M rows that exist */
    return f < 0 ? 0 : (f > s.M ? s.M : f);
}
__device__ __forceinline__ int group_count(const SpRowsSeg &s, int g) {
    if (s.offset) { int l = __ldcg(s.offset + g + 1); l = l > s.M ? s.M : l; const int c = l - group_first(s, g); return c < 0 ? 0 : c; }
    if (!s.count) return s.M;
    const int c = __ldcg(s.count + g);
    return c > s.M ? s.M : c;
}
__device__ __forceinline__ int unit_log(int cnt, int many) { return cnt > many ? 4 : 2; }      /* log2 of the tokens of a group's units at most */
__device__ __forceinline__ int units_of(int cnt, int log) { return (cnt + (1 << log) - 1) >> log; }
__device__ Unit locate(const RowsArgs &a, const Plan &p, int u) {
    Unit r{};
    r.seg = u >= p.total[0] ? 1 : 0;
    const SpRowsSeg &s = a.seg[r.seg];
    u -= r.seg ? p.total[0] : 0;
    const int *st = p.start[r.seg];
    int lo = 0, hi = s.groups - 1;                          /* the last group that starts at or before u: never an empty one */
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (st[mid] <= u) lo = mid; else hi = mid - 1; }
    r.grp = lo;
    const int cnt = r.seg && p.count ? p.count[lo] : group_count(s, lo), log = unit_log(cnt, r.seg ? a.many[1] : a.many[0]), nr = units_of(cnt, log), k = u - st[lo];
    r.tile = k / nr;
    r.t0 = (k - r.tile * nr) << log;
    r.nt = cnt - r.t0 < 1 << log ? cnt - r.t0 : 1 << log;
    return r;
}

/* out of line, for the units after the first: rare, and no code of it in the loops of the copy warps */
__device__ __noinline__ UnitWord locate_out(const RowsArgs &a, const Plan &p, int u) { return pack(locate(a, p, u)); }

/* ---------------------------------------------------------------- the dots of one warp: 16 rows x four tokens */
/* W = 1: one chunk x four tokens fill the eight columns of B. W = 2: two neighbouring chunks (a group) x two tokens; lane q of
 * a row reads two words, one per MMA, and column 2 u + h takes half h of the (token, chunk) u. Either way lane q's C registers
 * hold both block sums of one (row, token, chunk) for two rows. */
extern __shared__ unsigned char sm_raw[];
/* loads by offset: pointers that are chosen at run time would become generic loads, which take the long way */
template <class T> __device__ __forceinline__ T lds(unsigned at) { return *reinterpret_cast<const T *>(sm_raw + at); }
struct Frag {
    unsigned w0, w1;                   /* (offsets in shared memory) this lane's two rows, at its words of a piece */
    unsigned s0, s1;                   /* their block scales, at the lane's chunk of a group */
    unsigned b;                        /* the lane's bytes of its column's token and half, or zeros */
    unsigned sx;                       /* block scales of the lane's token, at its chunk of a group */
    int n32, row, piece;               /* row % 8; the chunk of a group whose words the lane reads */
};
/* group slots r, r + 4, ... (32 / W of them, groups s + 32 / W i of each), added as the tree adds them: s and s + 16 (chunks),
 * then + 8, then, W = 1, + 4. Slots from chunk 4 * NJ on are known to be empty (NJ even). Chunk c of a row is piece c % 8 of
 * slice c / 8 (SL bytes apart), swizzled by the row. */
template <int W, int SL, int NI, int NJ = 8>
__device__ __forceinline__ float2 class_sum(const Frag &f, int r) {
    const unsigned p = (unsigned)((W * r + f.piece) ^ f.row) << 4;
    const unsigned w0e = f.w0 + p, w0o = f.w0 + (p ^ 64u), w1e = f.w1 + p, w1o = f.w1 + (p ^ 64u);
    const unsigned b0 = f.b + 32 * W * r, s0 = f.s0 + 2 * W * r, s1 = f.s1 + 2 * W * r, x0 = f.sx + 8 * W * r;
    auto slot = [&](int j) {
        float2 acc = make_float2(0.0f, 0.0f);
        if (j * W >= NJ) return acc;
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const int c = 4 * W * j + 32 * i, at = ((W * j >> 1) + 4 * i) * SL;      /* c: beyond W r */
            if (i + 1 < NI || W * r + c < f.n32) {          /* warp-uniform */
                const float2 s2 = lds<float2>(x0 + 8 * c);
                const float ws0 = h2f(lds<unsigned short>(s0 + 2 * c)), ws1 = h2f(lds<unsigned short>(s1 + 2 * c));
                int d[4];
                if (W == 1) {
                    const unsigned u0 = lds<unsigned>((j & 1 ? w0o : w0e) + at), u1 = lds<unsigned>((j & 1 ? w1o : w1e) + at);
                    const uint2 b = lds<uint2>(b0 + 32 * c);
                    mma_s8(d, (u0 << 4) & 0xF0F0F0F0u, (u1 << 4) & 0xF0F0F0F0u, u0 & 0xF0F0F0F0u, u1 & 0xF0F0F0F0u, b.x, b.y, kMagic);
                } else {
                    const uint2 u0 = lds<uint2>(w0e + at), u1 = lds<uint2>(w1e + at);
                    const uint4 b = lds<uint4>(b0 + 32 * c);
                    mma_s8(d, (u0.x << 4) & 0xF0F0F0F0u, (u1.x << 4) & 0xF0F0F0F0u, u0.x & 0xF0F0F0F0u, u1.x & 0xF0F0F0F0u, b.x, b.y, kMagic);
                    mma_s8_add(d, (u0.y << 4) & 0xF0F0F0F0u, (u1.y << 4) & 0xF0F0F0F0u, u0.y & 0xF0F0F0F0u, u1.y & 0xF0F0F0F0u, b.z, b.w);
                }
                const float2 g = magic_to_float2(d[0], d[1]), h = magic_to_float2(d[2], d[3]);
                acc.x = __fmaf_rn(ws0, __fmaf_rn(g.x, s2.x, __fmul_rn(g.y, s2.y)), acc.x);
                acc.y = __fmaf_rn(ws1, __fmaf_rn(h.x, s2.x, __fmul_rn(h.y, s2.y)), acc.y);
            }
        }
        return acc;
    };
    auto add = [](float2 p, float2 q) { return make_float2(p.x + q.x, p.y + q.y); };
    if (W == 2) { const float2 a = add(slot(0), slot(2)); return add(a, add(slot(1), slot(3))); }
    float2 a = add(slot(0), slot(4)); a = add(a, add(slot(2), slot(6)));
    float2 b = add(slot(1), slot(5)); b = add(b, add(slot(3), slot(7)));
    return add(a, b);
}
template <int W, int SL>
__device__ __forceinline__ float2 class_sum_n(const Frag &f, int r) {
    if (f.n32 <= 32) return class_sum<W, SL, 1>(f, r);
    if (f.n32 <= 64) return class_sum<W, SL, 2>(f, r);
    if (f.n32 <= 96) return class_sum<W, SL, 3>(f, r);
    return class_sum<W, SL, 4>(f, r);
}
/* rows of up to 32 chunks: all four classes by one warp, (0 + 2) + (1 + 3), then the two chunks of a group (lanes q, q ^ 1) */
template <int W, int SL>
__device__ __forceinline__ float2 row_sum(const Frag &f) {
    float2 v = make_float2(0.0f, 0.0f), o = v;
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        const int r = k == 1 ? 2 : k == 2 ? 1 : k;
        const float2 c = f.n32 <= 8 ? class_sum<W, SL, 1, 2>(f, r) : f.n32 <= 16 ? class_sum<W, SL, 1, 4>(f, r) : f.n32 <= 24 ? class_sum<W, SL, 1, 6>(f, r) : class_sum<W, SL, 1, 8>(f, r);
        if (k == 0 || k == 2) o = c;
        else { o.x += c.x; o.y += c.y; if (k == 1) v = o; else { v.x += o.x; v.y += o.y; } }
    }
    if (W == 2) { v.x += __shfl_xor_sync(0xffffffffu, v.x, 1); v.y += __shfl_xor_sync(0xffffffffu, v.y, 1); }
    return v;
}

/* ---------------------------------------------------------------- the kernel
 * Warps: teams x 8 that multiply, one that copies weights, one per team that copies activations. */
struct Batch { int seg, tile, flags, item[kTok], pad; };     /* up to four tokens of a unit; flags: 1 = the unit's first, 2 = its last, 4 = the team is done, 8 = more than two tokens */

template <bool PAIR, int W>
__global__ void __launch_bounds__(kMaxTeams *kTeamThreads + 96, 1) k_rows(const __grid_constant__ RowsArgs a) {
    unsigned char *const sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
    __shared__ unsigned long long bars[(1 + kMaxTeams) * kMaxStages + 6 * kMaxTeams];
    __shared__ int abort_s;
    __shared__ Batch batch_s[kMaxTeams][2];
    __shared__ float part_s[kMaxTeams][2][4 * 2 * 16 * kTok];
    __shared__ UnitWord units_s[kUnits], later_s[32];
    __shared__ int start_s[1 + 1024], total_s[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    volatile int *abort_flag = &abort_s;
    const uint32_t bar0 = smem_u32(bars);
    /* weight stages. A stage may serve the teams in turn, and its fills land in any order: each team waits on barriers that count
     * its own fills only (on a shared one, a team could take the phase before the other's fill for its own) */
    auto full = [&](int team, int s) { return bar0 + 8u * (kMaxStages * (1 + team) + s); };
    auto empty = [&](int s) { return bar0 + 8u * s; };
    constexpr int kActBars = (1 + kMaxTeams) * kMaxStages;
    auto afull = [&](int team, int b) { return bar0 + 8u * (kActBars + 6 * team + b); };      /* a team's two buffers of activations */
    auto aempty = [&](int team, int b) { return bar0 + 8u * (kActBars + 6 * team + 2 + b); };
    auto sums = [&](int team, int b) { return bar0 + 8u * (kActBars + 6 * team + 4 + b); };      /* and of sums: all eight warps' are there */
    if (tid == 0) {
        for (int s = 0; s < a.stages; s++) {
            for (int t = 0; t < a.teams; t++) mbar_init(full(t, s), 1);
            mbar_init(empty(s), kTeamWarps);
        }
        for (int t = 0; t < a.teams; t++)
            for (int b = 0; b < 2; b++) {
                mbar_init(afull(t, b), 1); mbar_init(aempty(t, b), kTeamWarps); mbar_init(sums(t, b), kTeamWarps);
            }
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    unsigned char *const zeros = sm + (unsigned)a.stages * a.stage_bytes + (unsigned)a.teams * 2u * a.act_bytes;
    for (unsigned i = tid; i < a.zero_bytes / 16; i += blockDim.x) reinterpret_cast<uint4 *>(zeros)[i] = make_uint4(0u, 0u, 0u, 0u);
    sp_pdl_wait();
    sp_pdl_next();
    /* first unit of every group, per segment (segment 0 is the only one or has one group) */
    int *const count_s = reinterpret_cast<int *>(part_s);     /* until the teams start */
    if (warp == 0) {
        int at = 0;
        for (int k = 0; k < 2; k++) {
            int run = 0;
            if (k < a.nseg) {
                const SpRowsSeg &s = a.seg[k];
                for (int g0 = 0; g0 < s.groups; g0 += 32) {
                    const int g = g0 + lane;
                    const int cnt = g < s.groups ? group_count(s, g) : 0, n = a.geo[k].tiles * units_of(cnt, unit_log(cnt, k ? a.many[1] : a.many[0]));
                    if (k == 1 && g < s.groups) count_s[g] = cnt;
                    int v = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += t; }
                    if (g < s.groups) start_s[at + g] = run + v - n;
                    run += __shfl_sync(0xffffffffu, v, 31);
                }
                at += s.groups;
            }
            if (lane == 0) total_s[k] = run;
        }
    }
    __syncthreads();
    Plan plan;
    plan.start[0] = start_s; plan.start[1] = start_s + a.seg[0].groups; plan.total[0] = total_s[0]; plan.total[1] = total_s[1]; plan.count = count_s;
    const int total = plan.total[0] + plan.total[1], G = gridDim.x;
    for (int i = tid; i < kUnits && (int)blockIdx.x + i * G < total; i += blockDim.x) units_s[i] = pack(locate(a, plan, blockIdx.x + i * G));
    plan.count = nullptr;
    __syncthreads();
    const int mine = total > (int)blockIdx.x ? (total - blockIdx.x + G - 1) / G : 0;
    /* units beyond the table: a warp finds its next 32 at once, a lane each. One after the other, 274 tokens of E 1344, 160 experts, 7
     * each, FFE 1472 (300 units a CTA) took 640 us a layer, 509 so; 256 tokens of E 2816, 128 experts, 8 each, FFE 704 493, 467 so. The
     * copy warps' loops over the table stay free of it (one loop for both: 1% at 32 and 64 tokens). */
    auto later = [&](int i) { return i < mine ? locate_out(a, plan, blockIdx.x + i * G) : UnitWord{0u, 0}; };
    const uint32_t sbase = smem_u32(sm);
    bool failed = false;

    if (warp == a.teams * kTeamWarps) {
        /* ---------------- weights */
        int s = 0, ph = 0;
        auto issue = [&](const Unit &u, int i) {
            const SpRowsSeg &sg = a.seg[u.seg];
            const SegGeo &ge = a.geo[u.seg];
            const int per = PAIR ? 16 : 16 * ge.mt_n, r0 = u.tile * per, nr = sg.rows - r0 < per ? sg.rows - r0 : per;
            const uint32_t dst = sbase + (unsigned)s * a.stage_bytes, sdst = dst + ge.scale_off, bar = full(i % a.teams, s);
            const int row = (int)((long long)u.grp * sg.rows_per_group) + r0;
            const unsigned sbytes = (unsigned)nr * ge.sb;
            const unsigned char *const ssrc = reinterpret_cast<const unsigned char *>(sg.bs) + (size_t)row * ge.sb;
            if (!mbar_wait(empty(s), ph ^ 1, abort_flag)) return false;
            mbar_expect_tx(bar, (PAIR ? 2 : 1) * (ge.box_bytes + sbytes));       /* rows past the tensor arrive as zeros */
            box_g2s(dst, &a.codes[u.seg][0], row, bar);
            if (PAIR) {
                box_g2s(dst + ge.box_bytes, &a.codes[u.seg][1], row + sg.up_off, bar);
                bulk_g2s(sdst + 16 * ge.sb, reinterpret_cast<const unsigned char *>(sg.ubs) + (size_t)(row + sg.up_off) * ge.sb, sbytes, bar);
            }
            bulk_g2s(sdst, ssrc, sbytes, bar);
            if (++s == a.stages) { s = 0; ph ^= 1; }
            return true;
        };
        const int table = mine < kUnits ? mine : kUnits;
        if (lane == 0)
            for (int i = 0; i < table; i++)
                if (!issue(unpack(units_s[i]), i)) { failed = true; break; }
        for (int i0 = kUnits; i0 < mine; i0 += 32) {
            __syncwarp();                                   /* lane 0 has read the words */
            if (__shfl_sync(0xffffffffu, failed, 0)) break;
            later_s[lane] = later(i0 + lane);
            __syncwarp();
            if (lane == 0)
                for (int i = i0; i < mine && i < i0 + 32; i++)
                    if (!issue(unpack(later_s[i - i0]), i)) { failed = true; break; }
        }
        __syncwarp();
    } else if (warp > a.teams * kTeamWarps) {
        /* ---------------- activations of one team: four tokens ahead of it, one lane per token */
        const int team = warp - a.teams * kTeamWarps - 1;
        const uint32_t abase = sbase + (unsigned)a.stages * a.stage_bytes + (unsigned)team * 2u * a.act_bytes;
        int n = 0, nl = 0;
        UnitWord ahead{0u, 0};
        for (int i = team; i < mine && !failed; i += a.teams) {
            UnitWord w;
            if (i < kUnits) w = units_s[i];
            else {
                if ((nl & 31) == 0) ahead = later(i + lane * a.teams);
                w.w = __shfl_sync(0xffffffffu, ahead.w, nl & 31); w.t0 = __shfl_sync(0xffffffffu, ahead.t0, nl & 31);
                nl++;
            }
            const Unit u = unpack(w);
            const SpRowsSeg &s = a.seg[u.seg];
            const SegGeo &ge = a.geo[u.seg];
            const int first = group_first(s, u.grp) + u.t0;
            for (int b = 0; b < u.nt; b += kTok, n++) {
                int item = -1, arow = 0;
                if (lane < kTok && b + lane < u.nt) {
                    const int at = first + b + lane;
                    if (s.offset) { item = s.index ? __ldcg(s.index + at) : at; arow = s.act_index ? __ldcg(s.act_index + at) : item; }
                    else { item = s.list ? __ldcg(s.list + (size_t)u.grp * s.list_stride + at) : at; arow = item; }
                    if (!s.act_index && s.act_div > 1) arow /= s.act_div;
                }
                const int buf = n & 1, have = u.nt - b < kTok ? u.nt - b : kTok;
                if (!mbar_wait(aempty(team, buf), ((n >> 1) & 1) ^ 1, abort_flag)) { failed = true; break; }
                Batch *d = &batch_s[team][buf];
                if (lane < kTok) d->item[lane] = item;
                if (lane == 0) { d->seg = u.seg; d->tile = u.tile; d->flags = (b == 0 ? 1 : 0) | (b + kTok >= u.nt ? 2 : 0) | (have > 2 ? 8 : 0); }
                __syncwarp();
                if (lane == 0) mbar_expect_tx(afull(team, buf), (unsigned)have * (unsigned)sp_act_pitch(s.in));        /* its arrival also publishes the descriptor */
                __syncwarp();
                if (item >= 0)
                    bulk_g2s(abase + buf * a.act_bytes + lane * ge.ast, s.act + (size_t)arow * sp_act_pitch(s.in), (unsigned)sp_act_pitch(s.in), afull(team, buf));
            }
        }
        if (!failed) {                                      /* one more descriptor: nothing left */
            const int buf = n & 1;
            if (!mbar_wait(aempty(team, buf), ((n >> 1) & 1) ^ 1, abort_flag)) failed = true;
            else if (lane == 0) {
                batch_s[team][buf].flags = 4;
                mbar_arrive(afull(team, buf));
            }
        }
    } else {
        /* ---------------- a team: units team, team + teams, ... of this CTA, four tokens at a time */
        const int team = warp / kTeamWarps, tw = warp % kTeamWarps, gq = lane >> 2, q = lane & 3;
        const unsigned char *const aptr = sm + (unsigned)a.stages * a.stage_bytes + (unsigned)team * 2u * a.act_bytes;
        int s = team % a.stages;
        unsigned phs = 0, psum = 0;                         /* bit s: parity of this team's next use of stage s; bit b: of buffer b of sums (pairs: of every batch) */
        Frag f;
        /* lanes whose 8-byte loads share a wavefront (W = 2) take rows whose pieces differ by more than the group's two */
        f.row = W == 1 ? gq : (gq & 1) << 2 | (gq & 2) | gq >> 2;
        f.piece = W == 1 ? 0 : q >> 1;
        const int cs = W == 1 ? 0 : q & 1, row = f.row;     /* cs: the chunk of a group in the lane's C registers */
        const bool bvalid = W == 1 ? (q >> 1) == (gq & 1) : q == (gq & 3);
        const int btok = W == 1 ? gq >> 1 : gq >> 2, ctok = W == 1 ? q : q >> 1;
        const unsigned z = (unsigned)(zeros - sm_raw) + (W == 1 ? (gq < 4 ? 64 : 0) + 8 * q : 96);      /* on banks the other lanes of the wavefront do not use */
        const int wo = W == 1 ? 4 * q : 8 * (q & 1), bo = (W == 1 ? 8 : 16) * q;
        for (int n = 0;; n++) {
            const int buf = n & 1;
            if (!mbar_wait(afull(team, buf), (n >> 1) & 1, abort_flag)) { failed = true; break; }
            const Batch &bt = batch_s[team][buf];
            const int flags = bt.flags;
            if (flags & 4) break;
            const int sgi = bt.seg, tile = bt.tile;
            const SpRowsSeg &sg = a.seg[sgi];
            const SegGeo &ge = a.geo[sgi];
            if ((flags & 1) && !mbar_wait(full(team, s), phs >> s & 1u, abort_flag)) { failed = true; break; }
            const int mt_n = PAIR ? 2 : ge.mt_n, mt = mt_n == 8 ? tw : tw >> 2, r0 = tile * 16 * mt_n;
            const unsigned codes = (unsigned)(sm - sm_raw) + (unsigned)s * a.stage_bytes, scales = codes + ge.scale_off, act = (unsigned)(aptr - sm_raw) + buf * a.act_bytes;
            if (PAIR) { f.w0 = codes + (mt * 8 + row) * 128 + wo; f.w1 = f.w0 + ge.box_bytes; f.s0 = scales + (mt * 8 + row) * ge.sb + 2 * cs; f.s1 = f.s0 + 16 * ge.sb; }      /* gate rows, then the up rows */
            else { f.w0 = codes + (mt * 16 + row) * 128 + wo; f.w1 = f.w0 + 8 * 128; f.s0 = scales + (mt * 16 + row) * ge.sb + 2 * cs; f.s1 = f.s0 + 8 * ge.sb; }
            f.n32 = ge.n32;
            const bool many = W == 2 && (flags & 8);        /* two pairs of tokens */
            auto tokens = [&](int first) {                  /* point the fragment at the W = 1: four, 2: two tokens from `first` */
                __syncwarp();                               /* the MMAs take the whole warp; a wait or the last tokens' stores may have split it */
                f.b = bvalid ? act + (first + btok) * ge.ast + bo : z;
                f.sx = act + (first + ctok) * ge.ast + sg.in + 8 * cs;
            };
            auto release = [&] {                            /* the stage, once the warp has read it for the last time; its lanes meet */
                __syncwarp();
                if (flags & 2) {
                    mbar_arrive_lane0(empty(s), lane);
                    phs ^= 1u << s;
                    s += a.teams;
                    while (s >= a.stages) s -= a.stages;
                }
            };
            if (!PAIR && mt_n == 8) {
                if (r0 + mt * 16 < sg.rows) {
#pragma unroll 1
                    for (int first = 0; first < (many ? 4 : 2); first += 4 / W) {
                        tokens(first);
                        const float2 v = row_sum<W, 128 * 128>(f);
                        const int it = bt.item[first + ctok];
                        if (it >= 0 && cs == 0) {
                            float *out = sg.out_f + (size_t)it * sg.out_stride + r0 + mt * 16 + row;
                            out[0] = v.x; out[8] = v.y;
                        }
                    }
                }
                release();
            } else {
                /* the eight warps: two 16-row tiles x four classes, or (W = 2, more than two tokens) two tiles x two pairs of
                 * tokens x two pairs of classes. part: [class sums left][tile][row][token] */
                float *part = part_s[team][buf];
                constexpr int SL = PAIR ? 16 * 128 : 32 * 128;
                const int T = W == 1 || many ? 4 : 2;
                if (PAIR || r0 + mt * 16 < sg.rows) {
                    int r = many ? tw & 1 : tw & 3;
                    tokens(many ? tw & 2 : 0);
                    float *p = part + (((W * r + cs) * 2 + mt) * 16 + row) * T + (many ? tw & 2 : 0) + ctok;
                    float2 v = make_float2(0.0f, 0.0f);
                    if (W == 1) v = class_sum_n<W, SL>(f, r);
                    else {
#pragma unroll 1
                        for (;; r += 2) {
                            const float2 c = class_sum_n<W, SL>(f, r);
                            if (r >= 2 && many) { v.x += c.x; v.y += c.y; break; }
                            v = c;
                            if (!many) break;
                        }
                    }
                    p[0] = v.x; p[8 * T] = v.y;
                }
                release();
                /* Two warps (gate|up) or one per token finish the sums, other ones each time, and only they wait for the rest, which is
                 * at its next tokens meanwhile: a warp loses the time of one finish in four (or two) times. The other buffer of sums
                 * and the other barrier serve those next tokens; the buffer's next use but one waits for this one's end (aempty). The
                 * wait gives up when a warp of the team did, whose sums never come (on named barriers, which cannot, the give-up path
                 * would have to arrive for others; 64 tokens take 158.5 us a layer either way, 512 tokens 866 so, 859 on those). */
                const uint32_t par = PAIR ? (uint32_t)(n >> 1) & 1u : psum >> buf & 1u;
                if (!PAIR) psum ^= 1u << buf;
                mbar_arrive_lane0(sums(team, buf), lane);
                auto total_of = [&](int m, int rw, int t) {                 /* the last levels of the tree */
                    const float *p = part + (m * 16 + rw) * T + t;
                    const int k = 32 * T;
                    if (T == 4) return (p[0] + p[2 * k]) + (p[k] + p[3 * k]);
                    return ((p[0] + p[4 * k]) + (p[2 * k] + p[6 * k])) + ((p[k] + p[5 * k]) + (p[3 * k] + p[7 * k]));
                };
                if (PAIR) {
                    const int w0 = 2 * (n & 3);
                    if (tw == w0 || (tw == w0 + 1 && T == 4)) {
                        if (!mbar_wait_out(sums(team, buf), par, abort_flag)) { failed = true; break; }
                        __syncwarp();                       /* the quantisation takes the whole warp */
                        const int idx = (tw - w0) * 32 + lane, t = idx >> 4, col = idx & 15;
                        const float h = gelu_mul(total_of(col >> 3, col & 7, t), total_of(col >> 3, (col & 7) + 8, t));
                        const int it = bt.item[t] < 0 ? 0 : bt.item[t];
                        unsigned char *o = sg.out_act + (size_t)it * sp_act_pitch(sg.rows);
                        quant_elem16(h, bt.item[t] >= 0, reinterpret_cast<signed char *>(o) + tile * 16, reinterpret_cast<float *>(o + sg.rows) + tile);
                    }
                } else {
                    const int t = tw - 4 * (n & 1);
                    if (t >= 0 && t < T) {
                        if (!mbar_wait_out(sums(team, buf), par, abort_flag)) { failed = true; break; }
                        const int it = bt.item[t];
                        if (it >= 0 && r0 + lane < sg.rows) sg.out_f[(size_t)it * sg.out_stride + r0 + lane] = total_of(lane >> 4, lane & 15, t);
                    }
                }
            }
            __syncwarp();
            mbar_arrive_lane0(aempty(team, buf), lane);
        }
    }
    if (failed) {
        if (lane == 0) atomicExch(a.status, SP_KERR_BARRIER_TIMEOUT);
        __nanosleep(100000);                                /* let copies in flight land before the CTA leaves */
    }
}

/* the codes of a tensor as [128-byte slice][row][128 bytes]: the last slice of a row may reach into the next row (or into the
 * scales that follow the tensor in the arena); such chunks are not multiplied */
cudaError_t codes_map(const uint8_t *codes, const SpRowsSeg &s, const SegGeo &g, bool pair, CUtensorMap *m) {
    EncodeTiledFn fn = nullptr;
    const cudaError_t e = encode_tiled_fn(&fn);
    if (e != cudaSuccess) return e;
    const size_t rows = s.rows_per_group ? (size_t)s.groups * (size_t)s.rows_per_group : (size_t)s.rows;
    const cuuint64_t rb = (cuuint64_t)s.in / 2, slices = (rb + 127) / 128;
    const cuuint64_t dims[3] = {128, (cuuint64_t)rows, slices}, strides[2] = {rb, 128};
    const cuuint32_t box[3] = {128, (cuuint32_t)box_rows(g, pair), (cuuint32_t)slices}, estr[3] = {1, 1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t *>(codes), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
constexpr size_t kSmemLimit = 227 * 1024 - 14 * 1024;      /* dynamic part: the static arrays of the kernel take 13.3 KB */

}  // namespace

cudaError_t sp_rows_prepare() {
    for (const auto k : {k_rows<true, 1>, k_rows<true, 2>, k_rows<false, 1>, k_rows<false, 2>}) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t sp_rows_launch(const SpRowsSeg *seg, int nseg, bool pair, long long items, int *status, cudaStream_t st, int *nl) {
    RowsArgs a{};
    cudaError_t e = cudaSuccess;
    a.nseg = nseg; a.status = status;
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    /* two chunks x two tokens per MMA while most chosen experts have one or two tokens and the rows are whole groups. Us a layer
     * with one / two chunks, the line at one item per expert: E 2816, 128 experts, 8 each, FFE 704, line at 16 tokens: 42.7 / 39.6
     * at 2, 56.3 / 54.0 at 5, 77.7 / 75.7 at 12, 88.7 / 88.4 at 16, 96.7 / 97.0 at 20, 112 / 123 at 32, 162 / 197 at 64. E 2048, 64
     * experts, 6 each, FFE 1408, line at 10: 66.3 / 56.6 at 6, 85.1 / 71.9 at 10, 89.8 / 77.8 at 12, 101 / 92.4 at 16, 115 / 114 at 24.
     * E 1024, 32 experts, 4 each, FFE 512, line at 8: 21.5 / 20.5 at 2, 23.4 / 24.2 at 4, 28.0 / 29.0 at 8, 29.1 / 30.7 at 10. The line
     * is right for the first; the longer down rows of the second would move it to twice as many tokens, the short ones of the
     * third to a quarter of them. */
    bool whole = items <= (seg[nseg - 1].owners ? seg[nseg - 1].owners : seg[nseg - 1].groups);
    /* Small units all cost about the same: with up to 16 tokens to a unit, one of the shared expert held its stage for a third of
     * the launch at 16 tokens and kept the other team waiting. What small ones fetch again comes from L2, until that is what
     * bounds them. Us a layer of E 2816, 128 experts, 8 each, units of 16 / 8 / 4 tokens: 54.4 / 54.5 / 52.8 at 5 tokens, 92.2 / 88.5 /
     * 86.6 at 16, 120 / 119 / 113 at 32, 176 / 174 / 160 at 64; of 16 / 4: 238 / 222 at 100, 412 / 395 at 200, 550 / 501 at 256, 772 / 760 at
     * 400 (321: 693 / 623), 901 / 967 at 512, 1677 / 1870 at 1024: the line is at 384 tokens, 24 items to an expert on average
     * (E 2048, 64 experts, 6 each: 869 / 746 at 24 items, 1029 / 1083 at 36; E 1024, 32 experts, 4 each: 121 / 103 at 24, 136 /
     * 128 at 32, where it could lie higher). Where the router sends most tokens to a few experts, those alone are above the
     * line: a group of more than 48 items has units of 16 whatever the average (a Zipf 1.2 router over 128 experts, units of 4 everywhere /
     * so: 242 / 237 at 128 tokens, 463 / 428 at 256, 687 / 613 at 384). 48, because units of both sizes side by side cost
     * more than they save while the counts only scatter about their average (384 tokens, 24 on average: a line of 24 per group 757,
     * of 48 721). And only where there would still be 16 units of that size to an SM: the few of a small launch end unevenly (60 experts, 7
     * each, E 2688, FFE 1088, Zipf, 49 tokens: 138 with units of 16, 124; 16 experts, 2 each, E 576, FFE 832, 113 tokens: 54, 49). Rows sorted for one rank's experts belong to fewer groups than there are, how many is not known here: their line
     * is 24 for each group by itself, with the same condition. */
    const bool few = items <= (long long)kFewItems * seg[nseg - 1].groups;
    for (int i = 0; i < nseg; i++) {
        a.seg[i] = seg[i];
        const long long units = (long long)seg_geo(seg[i], pair).tiles * (i + 1 < nseg ? seg[i].M : items) / 16;
        const int line = units >= kSmUnits * (long long)sms ? (seg[i].offset ? kFewItems : kManyItems) : 0x7fffffff;
        a.many[i] = !few && !seg[i].offset ? 0 : seg[i].groups > 1 ? line : 0x7fffffff;
        const SegGeo &g = a.geo[i] = seg_geo(seg[i], pair);
        const unsigned sb = up1024(g.scale_off + 16 * g.mt_n * g.sb), ab = kTok * g.ast;
        const unsigned zb = (unsigned)seg[i].in + 128;
        a.zero_bytes = zb > a.zero_bytes ? zb : a.zero_bytes;
        whole = whole && g.n32 % 2 == 0;
        a.stage_bytes = sb > a.stage_bytes ? sb : a.stage_bytes; a.act_bytes = ab > a.act_bytes ? ab : a.act_bytes;
    }
    /* two teams with three stages where they fit (one being filled while two are used), else one team with two */
    for (int i = 0; i < nseg; i++) {
        e = codes_map(seg[i].codes, seg[i], a.geo[i], pair, &a.codes[i][0]);
        if (e == cudaSuccess && pair) e = codes_map(seg[i].ucodes, seg[i], a.geo[i], pair, &a.codes[i][1]);
        if (e != cudaSuccess) return e;
    }
    a.teams = (size_t)3 * a.stage_bytes + 4 * (size_t)a.act_bytes + a.zero_bytes + 1024 <= kSmemLimit ? 2 : 1;
    const size_t acts = (size_t)a.teams * 2 * a.act_bytes + a.zero_bytes;
    a.stages = (int)((kSmemLimit - 1024 - acts) / a.stage_bytes);
    if (a.stages > kMaxStages) a.stages = kMaxStages;
    if (a.stages < 1) return cudaErrorInvalidValue;
    const unsigned threads = (unsigned)(a.teams * kTeamThreads + 32 + 32 * a.teams);
    const size_t smem = acts + (size_t)a.stages * a.stage_bytes + 1024;
    return sp_launch(pair ? whole ? k_rows<true, 2> : k_rows<true, 1> : whole ? k_rows<false, 2> : k_rows<false, 1>, dim3((unsigned)sms), threads, smem, st, nl, a);
}
