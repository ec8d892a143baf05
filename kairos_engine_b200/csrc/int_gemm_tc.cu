/* int_gemm_tc.cu — the reference's quantised PTX-MMA GEMM on tcgen05:
 *     C[m][n] (f16) = f16( float(sum_k A[m][k] * B[n][k]) * scale_a[m] * scale_b[n] )
 * int8 (or packed signed int4) operands, int32 accumulate, per-row x per-column fp32 scales.
 * Replaces sp_frob_matmul_q8_mma_tile / sp_frob_matmul_q4_mma_* (src/backends/cuda/ptx_mma.cuh:
 * 115-222, 268-353; ptx_mma_tile_int8.cuh:92-110; epilogue ptx_mma_tile_common.cuh:157-176), which
 * tile mma.sync m8n8k16 / m8n8k32 per warp. Here: tcgen05.mma kind::i8 (128 x NT x 32 per
 * instruction), both operands by TMA into 128-byte-swizzled K-major tiles, int32 accumulators in
 * tensor memory, the same epilogue arithmetic and operation order, so results are bit-identical to
 * the reference's.
 * A is [M][K], B is [N][K] (the tiled kernels' layout); K a multiple of 16.
 * Tile: MH x 128 rows of A x NT rows of B, k in stages of 128. What bounds it is moving operands: an MMA of 128 x NT x 32
 * reads 4 + NT/32 KB of shared memory, and each stage comes from L2 once. A tile of 256 x 256 (two MMAs share a B tile; its
 * accumulators fill tensor memory, so there is one set) takes 0.37 GB from L2 for 3072 x 8192 x 3072 and 4.1 GB for 8192^3
 * where 128 x 256 takes 0.66 and 6.6. Calls in a row, 256 x 256 / 128 x 256: 55.8 / 57.7 us, 442 / 501 us (at the power limit, where
 * the traffic saved becomes clock), 34 / 37 us at 2048 x 8192 x 2048, but about 66 / 62 us at 4096^3, where the second set of
 * accumulators hides the emptying. The tensor pipe is active 69 to 75% of the cycles an SM is active with 256 x 256, 72
 * to 80% with 128 x 256. Small problems take smaller tiles, to have one for every SM (pick_tile).
 * Packed int4 operands are unpacked on the way: sixteen warps read the packed rows and write the int8 tiles (the even
 * elements of every 8, then the odd ones, in both operands: an integer dot product does not see the order).
 * Warp roles: 0-7 epilogue (TMEM lane quadrant = warp % 4), 8 TMA, 9 MMA issue + TMEM allocation, 10-25 int4 unpack. Every
 * wait is bounded.
 */
#include <condition_variable>
#include <mutex>
#include "tc_common.cuh"
#include "../../include/sp_engine/moe_backend.h"

namespace {
using namespace sp_tc;

constexpr int kBKB = 128, kMaxDevices = 64, kEpiWarps = 8, kUnpWarps = 16;
template <int MH, int NT, bool PACKED> struct IgCfg {
    static constexpr int kStages = MH * 128 + NT >= 512 ? (PACKED ? 2 : 3) : MH * 128 + NT >= 384 ? (PACKED ? 3 : 4) : MH * 128 + NT >= 256 ? (PACKED ? 4 : 6) : 6, kBufs = MH * NT > 256 ? 1 : 2;
    static constexpr uint32_t kABytes = MH * 128 * 128, kBBytes = NT * 128, kStage = kABytes + kBBytes;
    static constexpr int kRaw = MH * 128 + NT >= 384 ? 3 : MH * 128 + NT >= 256 ? 5 : 6;      /* packed: stages of raw bytes */
    static constexpr int kUnits = 4 * (MH * 128 + NT);                                     /* packed: 16-byte pieces of a stage */
    static constexpr uint32_t kRawOff = kStages * kStage, kRawBytes = PACKED ? kUnits * 16 : 0;
    static constexpr uint32_t kBarOff = kRawOff + kRaw * kRawBytes, kSmem = kBarOff + 192 + 1024;
    static constexpr uint32_t kCols = MH * NT * kBufs < 128 ? 128 : MH * NT * kBufs;      /* TMEM columns, a power of two */
    static constexpr int kThreads = 32 * (kEpiWarps + 2 + (PACKED ? kUnpWarps : 0));
};

struct IgMaps { CUtensorMap a, b; };
struct IgArgs { const uint8_t *A, *B; const float *scale_a, *scale_b; __half *C; int M, K, N; int *status; };

/* 8 packed int4 (one word) -> the four even elements and the four odd ones as int8 */
__device__ __forceinline__ uint2 unpack_s4(uint32_t w) {
    const uint32_t e = w & 0x0F0F0F0Fu, o = (w >> 4) & 0x0F0F0F0Fu;
    return make_uint2(e | (e & 0x08080808u) * 30u, o | (o & 0x08080808u) * 30u);          /* bit 3 copied into bits 4-7 */
}

template <int MH, int NT, bool PACKED>
__global__ void __launch_bounds__(IgCfg<MH, NT, PACKED>::kThreads, 1) k_i8_gemm(const __grid_constant__ IgMaps maps, const IgArgs g) {
    using C = IgCfg<MH, NT, PACKED>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, M = g.M, K = g.K, N = g.N;
    const uint32_t bar0 = sbase + C::kBarOff;
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 48u + 8u * s; };
    auto tfull = [&](int b) { return bar0 + 96u + 8u * b; };
    auto tempty = [&](int b) { return bar0 + 112u + 8u * b; };
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + C::kBarOff + 128);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + C::kBarOff + 132);
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; s++) { mbar_init(full(s), PACKED ? kUnpWarps : 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(tfull(b), 1); mbar_init(tempty(b), kEpiWarps); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void *)tmem_slot)), "r"(C::kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    constexpr int TM = MH * 128;
    const int tn = (N + NT - 1) / NT, total = ((M + TM - 1) / TM) * tn, KB = (K + kBKB - 1) / kBKB;
    bool failed = false;

    if (warp == 8) {
        if (!PACKED && lane == 0) {
            int s = 0; uint32_t ph = 0;
            for (int w = blockIdx.x; w < total && !failed; w += gridDim.x) {
                const int m0 = (w / tn) * TM, n0 = (w % tn) * NT;
                for (int kb = 0; kb < KB; kb++) {
                    if (!mbar_wait(empty(s), ph ^ 1, abort_flag)) { failed = true; break; }
                    mbar_expect_tx(full(s), C::kStage);               /* rows or k beyond the matrices arrive as zeros */
                    const uint32_t dst = sbase + s * C::kStage;
                    tma_load_2d(dst, &maps.a, kb * kBKB, m0, full(s));
                    tma_load_2d(dst + C::kABytes, &maps.b, kb * kBKB, n0, full(s));
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
            }
            if (failed || *abort_flag) __nanosleep(100000);
        }
        __syncwarp();
    } else if (warp == 9) {
        /* s8 x s8 -> s32: c_format 2, a/b_format 1 (signed 8-bit), K-major both, N = NT, M = 128 */
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)NT >> 3) << 17) | ((128u >> 4) << 24);
        const bool leader = elect_one();
        int s = 0, lt = 0; uint32_t ph = 0;
        for (int w = blockIdx.x; w < total && !failed; w += gridDim.x, lt++) {
            const int b = lt % C::kBufs; const uint32_t bph = (lt / C::kBufs) & 1;
            if (!mbar_wait(tempty(b), bph ^ 1, abort_flag)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d0 = tmem + (uint32_t)(b * MH * NT);
            for (int kb = 0; kb < KB; kb++) {
                if (!mbar_wait(full(s), ph, abort_flag)) { failed = true; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (leader) {
                    const uint64_t a0 = make_desc(sbase + s * C::kStage), b0 = make_desc(sbase + s * C::kStage + C::kABytes);
#pragma unroll
                    for (int ks = 0; ks < kBKB / 32; ks++)
#pragma unroll
                        for (int h = 0; h < MH; h++)
                            umma_i8(d0 + h * NT, a0 + (uint64_t)(h * 1024 + ks * 2), b0 + (uint64_t)(ks * 2), idesc, (kb | ks) ? 1u : 0u);       /* in 16-byte units */
                    umma_commit(empty(s));
                    if (kb + 1 == KB) umma_commit(tfull(b));
                }
                __syncwarp();
                if (++s == C::kStages) { s = 0; ph ^= 1; }
            }
        }
    } else if (PACKED && warp >= 10) {
        /* packed rows -> int8 tiles. A thread takes 16-byte pieces u, u + 512, ... of a stage (four neighbours a row): they
         * travel kRaw - 1 stages ahead by asynchronous copies into a place of the thread's own (zeros past the edges) */
        constexpr int R = (C::kUnits + 32 * kUnpWarps - 1) / (32 * kUnpWarps);
        const int u0 = threadIdx.x - 320; const size_t pitch = (size_t)K / 2;
        const bool wide = (K & 31) == 0;                              /* rows on 16-byte boundaries, else on 8 */
        int s = 0, pw = blockIdx.x, pkb = 0, pslot = 0, uslot = 0; uint32_t ph = 0;
        auto fetch = [&]() {
            if (pw < total) {
                const int m0 = (pw / tn) * TM, n0 = (pw % tn) * NT;
#pragma unroll
                for (int q = 0; q < R; q++) {
                    const int u = u0 + 32 * kUnpWarps * q, r = u >> 2;
                    if (u < C::kUnits) {
                        const bool isa = r < TM; const int row = isa ? m0 + r : n0 + r - TM;
                        const bool ok = row < (isa ? M : N);
                        const size_t at = (size_t)pkb * 64 + 16 * (u & 3);
                        const uint8_t *p = (isa ? g.A : g.B) + (size_t)(ok ? row : 0) * pitch;
                        const int left = ok && at < pitch ? (int)(pitch - at < 16 ? pitch - at : 16) : 0;       /* bytes of the piece that exist: 0, 8 or 16 */
                        const uint32_t dst = sbase + C::kRawOff + pslot * C::kRawBytes + 16u * u;
                        if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(left ? p + at : p), "r"(left) : "memory");
                        else {
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(left ? p + at : p), "r"(left ? 8 : 0) : "memory");
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + 8u), "l"(left > 8 ? p + at + 8 : p), "r"(left > 8 ? 8 : 0) : "memory");
                        }
                    }
                }
                if (++pkb == KB) { pkb = 0; pw += gridDim.x; }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            pslot = pslot == C::kRaw - 1 ? 0 : pslot + 1;
        };
        for (int i = 0; i < C::kRaw - 1; i++) fetch();
        for (int w = blockIdx.x; w < total && !failed; w += gridDim.x)
            for (int kb = 0; kb < KB; kb++) {
                fetch();
                asm volatile("cp.async.wait_group %0;" ::"n"(C::kRaw - 1) : "memory");
                if (!mbar_wait(empty(s), ph ^ 1, abort_flag)) { failed = true; break; }
#pragma unroll
                for (int q = 0; q < R; q++) {
                    const int u = u0 + 32 * kUnpWarps * q, r = u >> 2, c = u & 3;
                    if (u < C::kUnits) {
                        const uint4 v = *reinterpret_cast<const uint4 *>(smem + C::kRawOff + uslot * C::kRawBytes + 16 * u);
                        unsigned char *row = smem + s * C::kStage + r * 128;       /* the B tile follows the A tile */
                        const uint2 a = unpack_s4(v.x), b = unpack_s4(v.y), d = unpack_s4(v.z), e = unpack_s4(v.w);
                        *reinterpret_cast<uint4 *>(row + (((2 * c) ^ (r & 7)) << 4)) = make_uint4(a.x, a.y, b.x, b.y);
                        *reinterpret_cast<uint4 *>(row + (((2 * c + 1) ^ (r & 7)) << 4)) = make_uint4(d.x, d.y, e.x, e.y);
                    }
                }
                uslot = uslot == C::kRaw - 1 ? 0 : uslot + 1;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                mbar_arrive_lane0(full(s), lane);
                if (++s == C::kStages) { s = 0; ph ^= 1; }
            }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < kEpiWarps) {
        /* epilogue (ptx_mma_tile_common.cuh:157-176): f16(float(acc) * sa[row] * sb[col]), left to right. The two warps of a
         * lane quadrant take alternate 16-column groups. */
        const int quad = warp & 3;
        const bool vec = (N & 7) == 0 && ((uintptr_t)g.C & 15) == 0;          /* every row on 16 bytes */
        int lt = 0;
        for (int w = blockIdx.x; w < total && !failed; w += gridDim.x, lt++) {
            const int n0 = (w % tn) * NT;
            const int b = lt % C::kBufs; const uint32_t bph = (lt / C::kBufs) & 1;
            if (!mbar_wait(tfull(b), bph, abort_flag)) { failed = true; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int h = 0; h < MH; h++) {
                const uint32_t t0 = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((b * MH + h) * NT);
                const int m = (w / tn) * TM + h * 128 + quad * 32 + lane; const bool rv = m < M;
                const float sa = rv ? __ldg(g.scale_a + m) : 0.0f;
                __half *crow = g.C + (size_t)(rv ? m : 0) * N;
#pragma unroll 1
                for (int c0 = (warp >> 2) * 16; c0 < NT; c0 += 32) {
                    const int nb = n0 + c0;
                    if (nb >= N) break;                                      /* warp-uniform */
                    uint32_t v[16];
                    tmem_ld16(t0 + c0, v);
                    const float mine = nb + (lane & 15) < N ? __ldg(g.scale_b + nb + (lane & 15)) : 0.0f;
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    __half o[16];
#pragma unroll
                    for (int n = 0; n < 16; n++)
                        o[n] = __float2half_rn(__fmul_rn(__fmul_rn(__int2float_rn((int)v[n]), sa), __shfl_sync(0xffffffffu, mine, n)));
                    if (rv) {
                        if (vec && nb + 16 <= N) {
                            *reinterpret_cast<uint4 *>(crow + nb) = *reinterpret_cast<const uint4 *>(o);
                            *reinterpret_cast<uint4 *>(crow + nb + 8) = *reinterpret_cast<const uint4 *>(o + 8);
                        } else {
#pragma unroll
                            for (int n = 0; n < 16; n++) if (nb + n < N) crow[nb + n] = o[n];
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty(b));
        }
    }
    if (failed && lane == 0) { *reinterpret_cast<volatile int *>(g.status) = SP_KERR_BARRIER_TIMEOUT; __threadfence_system(); }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) {
        if (*abort_flag) __nanosleep(100000);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kCols) : "memory");
    }
}

int ig_fail(int code, const char *msg) { sp_set_error(msg); return code; }

cudaError_t make_u8_map(EncodeTiledFn fn, CUtensorMap *m, const void *ptr, int K, int rows, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K};
    const cuuint32_t box[2] = {(cuuint32_t)kBKB, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

struct TileCfg { int mh, nt; };
constexpr TileCfg kTiles[4] = {{2, 256}, {1, 256}, {1, 128}, {1, 64}};
/* the tile with the shortest schedule: rounds of tiles over the SMs x shared-memory cycles of a stage (four MMA steps read
 * A and B, the stage is written once, 128 bytes a cycle; not less than the MMAs themselves) + the emptying of a tile */
int pick_tile(int M, int K, int N, int sms) {
    int best = 0; double best_t = 0.0;
    for (int i = 0; i < 4; i++) {
        const int mh = kTiles[i].mh, nt = kTiles[i].nt;
        const long long tiles = ((long long)(M + 128 * mh - 1) / (128 * mh)) * ((N + nt - 1) / nt);
        const double mma = 4.0 * mh * nt / 2, shared = 4.0 * mh * (4096 + 32 * nt) / 128 + (128.0 * mh + nt);
        const double t = (double)((tiles + sms - 1) / sms) * (((K + kBKB - 1) / kBKB) * (shared > mma ? shared : mma) + 6.0 * mh * nt);
        if (i == 0 || t < best_t) { best = i; best_t = t; }
    }
    return best;
}
/* Per device, made at first use there. words: page-locked, a kernel writes the one it is given when a bounded wait ran out.
 * Word 0 is the int8 entry's, which returns before its kernel runs; an int4 call has one of the others to itself, so that calls
 * from several threads do not read each other's verdict. */
constexpr int kWords = 64;
struct IgDevice { int *words; int sms; bool ready; unsigned long long taken; };
std::mutex g_mu;
std::condition_variable g_word_free;
IgDevice g_devices[kMaxDevices];
EncodeTiledFn g_encode = nullptr;

template <int MH, int NT, bool PACKED>
cudaError_t ig_prepare() { return cudaFuncSetAttribute(k_i8_gemm<MH, NT, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IgCfg<MH, NT, PACKED>::kSmem); }
template <bool PACKED>
cudaError_t ig_prepare_all() {
    cudaError_t e = ig_prepare<2, 256, PACKED>();
    if (e == cudaSuccess) e = ig_prepare<1, 256, PACKED>();
    if (e == cudaSuccess) e = ig_prepare<1, 128, PACKED>();
    return e == cudaSuccess ? ig_prepare<1, 64, PACKED>() : e;
}
template <int MH, int NT, bool PACKED>
void ig_launch(const IgMaps &maps, const IgArgs &g, int sms, cudaStream_t st) {
    const long long tiles = ((long long)(g.M + 128 * MH - 1) / (128 * MH)) * ((g.N + NT - 1) / NT);
    k_i8_gemm<MH, NT, PACKED><<<(unsigned)(tiles < sms ? tiles : sms), IgCfg<MH, NT, PACKED>::kThreads, IgCfg<MH, NT, PACKED>::kSmem, st>>>(maps, g);
}

int check_args(const void *A, const void *B, const float *sa, const float *sb, const uint16_t *C, int M, int K, int N) {
    if (!A || !B || !sa || !sb || !C) return ig_fail(SP_MOE_EBADARG, "quantised GEMM: NULL argument");
    if (M <= 0 || N <= 0 || K <= 0 || (K & 15)) return ig_fail(SP_MOE_EBADARG, "quantised GEMM: M, N, K must be positive and K a multiple of 16");
    return SP_MOE_OK;
}
/* the current device, ready for use */
int device_state(IgDevice **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return ig_fail(SP_MOE_ECUDA, "quantised GEMM: no CUDA device");
    if (dev < 0 || dev >= kMaxDevices) return ig_fail(SP_MOE_EUNSUPPORTED, "quantised GEMM: device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_encode && encode_tiled_fn(&g_encode) != cudaSuccess) return ig_fail(SP_MOE_EUNSUPPORTED, "quantised GEMM: cuTensorMapEncodeTiled is not available");
    IgDevice &d = g_devices[dev];
    if (!d.ready) {
        if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || ig_prepare_all<false>() != cudaSuccess || ig_prepare_all<true>() != cudaSuccess)
            return ig_fail(SP_MOE_ECUDA, "quantised GEMM: kernel attributes");
        if (!d.words && cudaMallocHost((void **)&d.words, kWords * sizeof(int)) != cudaSuccess) { d.words = nullptr; cudaGetLastError(); return ig_fail(SP_MOE_ECUDA, "quantised GEMM: status word allocation failed"); }
        for (int i = 0; i < kWords; i++) d.words[i] = 0;
        d.taken = 1;                                      /* word 0 */
        d.ready = true;
    }
    *out = &d;
    return SP_MOE_OK;
}

template <bool PACKED>
int enqueue(const IgDevice &dev, int *status, const void *A, const void *B, const float *sa, const float *sb, uint16_t *C, int M, int K, int N, cudaStream_t st) {
    const int sms = dev.sms;
    const int t = pick_tile(M, K, N, sms);
    IgMaps maps = {};
    if (!PACKED && (make_u8_map(g_encode, &maps.a, A, K, M, kTiles[t].mh * 128) != cudaSuccess || make_u8_map(g_encode, &maps.b, B, K, N, kTiles[t].nt) != cudaSuccess))
        return ig_fail(SP_MOE_EBADARG, "quantised GEMM: could not describe the operands to the TMA unit");
    const IgArgs g{(const uint8_t *)A, (const uint8_t *)B, sa, sb, reinterpret_cast<__half *>(C), M, K, N, status};
    switch (t) {
    case 0: ig_launch<2, 256, PACKED>(maps, g, sms, st); break;
    case 1: ig_launch<1, 256, PACKED>(maps, g, sms, st); break;
    case 2: ig_launch<1, 128, PACKED>(maps, g, sms, st); break;
    default: ig_launch<1, 64, PACKED>(maps, g, sms, st);
    }
    if (cudaGetLastError() != cudaSuccess) return ig_fail(SP_MOE_ECUDA, "quantised GEMM: kernel launch failed");
    return SP_MOE_OK;
}

}  // namespace

extern "C" int sp_frob_matmul_q8_dev(const int8_t *A_dev, const int8_t *B_dev, const float *scale_a_dev, const float *scale_b_dev,
                                     uint16_t *C_f16_dev, int M, int K, int N, void *stream) {
    int rc = check_args(A_dev, B_dev, scale_a_dev, scale_b_dev, C_f16_dev, M, K, N);
    if (rc == SP_MOE_OK && ((uintptr_t)A_dev | (uintptr_t)B_dev) & 15) rc = ig_fail(SP_MOE_EBADARG, "quantised GEMM: operand pointers must be 16-byte aligned");
    IgDevice *d = nullptr;
    if (rc == SP_MOE_OK) rc = device_state(&d);
    if (rc != SP_MOE_OK) return rc;
    volatile int *word = d->words;                        /* the kernel runs after this call has returned: what went wrong there is told to the next one */
    if (*word) { *word = 0; return ig_fail(SP_MOE_ECUDA, "sp_frob_matmul_q8_dev: in an earlier int8 call on this device a bounded wait inside the kernel ran out and its result is invalid; this call enqueued nothing"); }
    return enqueue<false>(*d, d->words, A_dev, B_dev, scale_a_dev, scale_b_dev, C_f16_dev, M, K, N, (cudaStream_t)stream);
}

extern "C" int sp_frob_matmul_q4_dev(const uint8_t *A_q4_dev, const uint8_t *B_q4_dev, const float *scale_a_dev, const float *scale_b_dev,
                                     uint16_t *C_f16_dev, int M, int K, int N, void *stream) {
    int rc = check_args(A_q4_dev, B_q4_dev, scale_a_dev, scale_b_dev, C_f16_dev, M, K, N);
    IgDevice *d = nullptr;
    if (rc == SP_MOE_OK) rc = device_state(&d);
    if (rc != SP_MOE_OK) return rc;
    /* the kernel copies pieces of 8 or 16 bytes: operands that start on another byte are moved first */
    cudaStream_t st = (cudaStream_t)stream;
    uint8_t *moved = nullptr;
    if (((uintptr_t)A_q4_dev | (uintptr_t)B_q4_dev) & 15) {
        const size_t na = (size_t)M * (K / 2), nb = (size_t)N * (K / 2), at = (na + 255) & ~(size_t)255;
        if (cudaMalloc((void **)&moved, at + nb) != cudaSuccess) { cudaGetLastError(); return ig_fail(SP_MOE_EBACKEND_OOM, "sp_frob_matmul_q4_dev: scratch allocation failed"); }
        if (cudaMemcpyAsync(moved, A_q4_dev, na, cudaMemcpyDeviceToDevice, st) != cudaSuccess || cudaMemcpyAsync(moved + at, B_q4_dev, nb, cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
            cudaStreamSynchronize(st); cudaFree(moved); cudaGetLastError();
            return ig_fail(SP_MOE_ECUDA, "sp_frob_matmul_q4_dev: copying the operands failed");
        }
        A_q4_dev = moved; B_q4_dev = moved + at;
    }
    int w = 0;
    {
        std::unique_lock<std::mutex> lk(g_mu);
        g_word_free.wait(lk, [&] { return ~d->taken != 0; });          /* every call that holds one is about to return */
        while (d->taken >> w & 1) w++;
        d->taken |= 1ull << w;
    }
    volatile int *word = d->words + w;
    *word = 0;
    rc = enqueue<true>(*d, d->words + w, A_q4_dev, B_q4_dev, scale_a_dev, scale_b_dev, C_f16_dev, M, K, N, st);
    /* this entry returns when the result is there, with the kernel's own verdict */
    if (cudaStreamSynchronize(st) != cudaSuccess && rc == SP_MOE_OK) rc = ig_fail(SP_MOE_ECUDA, "sp_frob_matmul_q4_dev: the stream reported an error");
    if (rc == SP_MOE_OK && *word) rc = ig_fail(SP_MOE_ECUDA, "quantised GEMM: a bounded wait inside the kernel ran out");
    {
        std::lock_guard<std::mutex> lk(g_mu);
        d->taken &= ~(1ull << w);
    }
    g_word_free.notify_all();                             /* the waiters may be of several devices */
    if (moved) cudaFree(moved);
    return rc;
}
