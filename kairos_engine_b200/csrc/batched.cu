/* batched.cu — the M > 1 paths of the MoE feed-forward layer: a few stream-ordered kernels per
 * layer with routing, bucketing and combine all on the device (no host round trip).
 *
 * Replaces g4_ffn_apply's expert-major batched branch (CF:8430-8965 of
 * src/backends/cuda/cuda_forward.cu): batched router prep + router GEMM, the D2H + host top-k +
 * host bucketing (CF:8483-8625), per-expert gather / GEMM / GELU split / GEMM / scatter-acc
 * (CF:8925-8965), and the recombine (CF:9014-9019).
 *
 * Two arithmetic flavours, the reference's AMMD switch (CF:8322-8324):
 *   decode  (per-token int8 activation quant + exact integer dots; what B sequential decode
 *            steps compute, CF:11737-11757) for small batches;
 *   prefill (w = code * f16 scale exactly, floating-point dot, fp32 accumulate; gemm_w,
 *            CF:13488-13518) for large ones.
 * Every (token, expert) pair is computed independently and the per-token combine walks the
 * experts in ascending id with acc = acc + w*out, so results do not depend on scheduling.
 */
#include "batched.cuh"
#include "prefill_tc.cuh"
#include "rows_mma.cuh"
#include "launch.cuh"
#include <cstdlib>
#include "../../include/sp_engine/moe_backend.h"

namespace {

struct BView {                 /* carved scratch */
    float *rin, *nx_f, *in_f, *logits, *cw, *hd, *dn, *h, *eo, *xa, *xb;
    unsigned char *nx_q, *in_q, *hd_q, *h_q;      /* quantised rows, sp_act_pitch apart */
    int *sel_asc, *count, *list, *pairpos, *ep_off;
    unsigned char *ep_q;      /* expert-parallel stage: quantised received rows, [max_rows] */
};

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }
constexpr int kSlices = SP_BATCHED_MAX_SLICES;     /* token slices of one layer that may be between route and finish at the same time */

template <class F>
size_t blayout(const SpDims &d, int Mx, int Rx, F place) {
    size_t o = 0; int id = 0;
    auto take = [&](size_t bytes) { place(id++, o); o = up256(o + bytes); };
    const size_t M = Mx, R = Rx, E = d.E, NE = d.NE, NU = d.NU, FFE = d.FFE, FFS = d.FFS;    /* R >= M * NU */
    take(4 * M * E); take(4 * M * E); take(4 * M * E); take(4 * M * NE); take(4 * M * NU);            /* rin nx_f in_f logits cw */
    take(4 * M * FFS); take(4 * M * E); take(4 * R * FFE); take(4 * M * NU * E);                     /* hd dn h eo */
    take(4 * M * E); take(4 * M * E);                                                               /* xa xb */
    take(M * sp_act_pitch(d.E)); take(M * sp_act_pitch(d.E)); take(M * sp_act_pitch(d.FFS)); take(R * sp_act_pitch(d.FFE));        /* q */
    take(4 * M * NU); take(4 * NE * kSlices); take(4 * NE * M);                                     /* sel_asc count list */
    take(R * sp_act_pitch(d.E));                                                                     /* ep_q */
    take(4 * M * NU); take(4 * (NE + 1) * kSlices);                                                 /* pairpos ep_off */
    return o;
}
BView bview(const SpDims &d, const SpBatchedScratch *s) {
    unsigned char *p[21];
    blayout(d, s->max_tokens, s->max_rows, [&](int id, size_t off) { p[id] = (unsigned char *)s->base + off; });
    BView v;
    v.rin = (float *)p[0]; v.nx_f = (float *)p[1]; v.in_f = (float *)p[2]; v.logits = (float *)p[3]; v.cw = (float *)p[4];
    v.hd = (float *)p[5]; v.dn = (float *)p[6]; v.h = (float *)p[7]; v.eo = (float *)p[8]; v.xa = (float *)p[9]; v.xb = (float *)p[10];
    v.nx_q = p[11]; v.in_q = p[12]; v.hd_q = p[13]; v.h_q = p[14];
    v.sel_asc = (int *)p[15]; v.count = (int *)p[16]; v.list = (int *)p[17];
    v.ep_q = p[18]; v.pairpos = (int *)p[19]; v.ep_off = (int *)p[20];
    return v;
}
/* The same scratch seen by token slice `slice` of a layer, whose first token is `t0`: everything the route stage
 * leaves for the finish stage (per-token and per-pair rows, the per-expert counters) moves to the slice's own
 * place, so several slices of one layer can be between route and finish at once (an expert-parallel run pipelines
 * them). What only the experts stage uses (h, the received rows' quantised copies) is shared: that stage runs one
 * slice at a time. */
BView bview_slice(const SpDims &d, const SpBatchedScratch *s, int t0, int slice) {
    BView v = bview(d, s);
    const size_t E = d.E, NE = d.NE, NU = d.NU, FFS = d.FFS, t = (size_t)t0;
    v.rin += t * E; v.nx_f += t * E; v.in_f += t * E; v.logits += t * NE; v.cw += t * NU; v.hd += t * FFS; v.dn += t * E; v.eo += t * NU * E;
    v.nx_q += t * sp_act_pitch(d.E); v.in_q += t * sp_act_pitch(d.E); v.hd_q += t * sp_act_pitch(d.FFS);
    v.sel_asc += t * NU; v.pairpos += t * NU; v.list += t * NE;
    v.count += (size_t)slice * NE; v.ep_off += (size_t)slice * (NE + 1);
    return v;
}

/* ---------------------------------------------------------------- device helpers */
__device__ __forceinline__ float rms_scale_from(double ss, int n, float eps) {
    const float ms = (float)(ss / (double)n);
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ms, eps)));
}
__device__ __forceinline__ float warp_tree(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
/* ---------------------------------------------------------------- K1/K7: everything a layer does per token
 * FIN: ordered combine and recombine of the layer that ends (CF:6071-6077, 9014-9019), which gives the residual y.
 * PREP: norms of y (or of x, without FIN) for the layer that begins (CF:8347, 8402-8404, 8425): the router's input and the
 * two experts' inputs as int8 blocks, fp32 rows, or fp16 hi/lo rows in the tensor-core GEMMs' k order.
 * One block per token, a thread takes two groups of four consecutive elements; what a thread needs is fetched before the
 * first dependent step, and what is left is three or four block-wide double sums in a row. Bound by their instructions (each
 * sum costs a warp some fifty, so few warps with more elements each), then by the pair rows it reads: see the figures at
 * launch_token. */
enum { kOutNone = 0, kOutInt8 = 1, kOutF32 = 2, kOutSplit = 3 };
struct TokArgs {
    const float *x;
    const float *dn, *eo, *cw; const int *pair_index; const float *post_ffw1, *post_ffw2, *post_ffw; float *y;       /* FIN */
    const float *ffn_norm, *pre_ffw2, *router_scale; float *rin; int *count;                                         /* PREP */
    unsigned char *nx_q, *in_q; float *nx_f, *in_f, *rows_f; __half *nx_hi, *nx_lo, *in_hi, *in_lo;
};
/* block-wide sums: shuffle tree per warp, then every warp adds the (at most 16) warps' sums by a second tree. `red` has 16
 * slots per sum, used once. */
template <int N>
__device__ __forceinline__ void block_sum(double (&a)[N], double *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; k++) a[k] += __shfl_down_sync(0xffffffffu, a[k], o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; k++) red[16 * k + warp] = a[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) a[k] = (lane & 15) < nw ? red[16 * k + (lane & 15)] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; k++) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
}
__device__ __forceinline__ double sumsq4(const float4 &f) { return ((double)f.x * f.x + (double)f.y * f.y) + ((double)f.z * f.z + (double)f.w * f.w); }
__device__ __forceinline__ float4 scale4(const float4 &f, float s, const float4 &w) {
    return make_float4(__fmul_rn(__fmul_rn(f.x, s), w.x), __fmul_rn(__fmul_rn(f.y, s), w.y), __fmul_rn(__fmul_rn(f.z, s), w.z), __fmul_rn(__fmul_rn(f.w, s), w.w));
}
/* four elements of a 16-block, four threads per block: quant_elem16's arithmetic and layout */
__device__ __forceinline__ void quant_quad(const float4 &f, bool ok, int i, unsigned char *act, int n) {
    float m = fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(f.z), fabsf(f.w)));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1)); m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    const float scale = m > 0.0f ? __fmul_rn(m, 1.0f / 127.0f) : 1.0f, inv = __fdiv_rn(1.0f, scale);
    auto one = [&](float v) { int t = __float2int_rn(__fmul_rn(v, inv)); t = t > 127 ? 127 : t; return t < -127 ? -127 : t; };
    const int a = one(f.x), b = one(f.y), c = one(f.z), d = one(f.w);
    if (ok) {
        unsigned char *g = act + 8 * (i >> 1) + 2 * (i & 1);        /* the even elements of a group of 8, then the odd ones */
        *reinterpret_cast<unsigned short *>(g) = (unsigned short)((a & 0xFF) | ((c & 0xFF) << 8));
        *reinterpret_cast<unsigned short *>(g + 4) = (unsigned short)((b & 0xFF) | ((d & 0xFF) << 8));
        if ((i & 3) == 0) reinterpret_cast<float *>(act + n)[i >> 2] = scale;
    }
}
/* four elements of a group of 8, two threads per group: fp16 hi and lo in the order 0,4,1,5,2,6,3,7; the lower thread
 * stores the group's hi, the upper its lo */
__device__ __forceinline__ void split_quad(const float4 &f, bool ok, int i, __half *hi, __half *lo) {
    const float v[4] = {f.x, f.y, f.z, f.w};
    unsigned h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const __half x = __float2half_rn(v[k]), y = __float2half_rn(__fsub_rn(v[k], __half2float(x)));
        h[k] = __half_as_ushort(x); l[k] = __half_as_ushort(y);
    }
    const bool up = i & 1;
    unsigned w[4];
    const unsigned s0 = up ? (h[0] | (h[1] << 16)) : (l[0] | (l[1] << 16)), s1 = up ? (h[2] | (h[3] << 16)) : (l[2] | (l[3] << 16));
    const unsigned r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
    const unsigned other[4] = {r0 & 0xFFFFu, r0 >> 16, r1 & 0xFFFFu, r1 >> 16};
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = up ? (other[k] | (l[k] << 16)) : (h[k] | (other[k] << 16));
    if (ok) *reinterpret_cast<uint4 *>((up ? lo : hi) + 8 * (i >> 1)) = make_uint4(w[0], w[1], w[2], w[3]);
}
/* FEW: at most one block per SM, so its latency counts: the norm weights are fetched while the previous kernel drains, all
 * pair rows at once. Otherwise three blocks (two of E above 3072) share an SM and the registers.
 * VEC: rows by 16-byte accesses. Without it (a caller's x, pair rows or y on some other float boundary) by single floats; the
 * handle's own vectors are aligned either way. */
template <bool FIN, int OUT, bool WIDE, bool FEW, bool VEC = true>
__global__ void __launch_bounds__(WIDE ? 512 : 384, FEW ? 1 : WIDE ? 2 : 3) k_b_token(SpDims d, TokArgs a) {
    constexpr int KB = FEW ? SP_MAX_NU : 4;
    __shared__ double red[3][32];
    const int t = blockIdx.x, E = d.E, NU = d.NU, T = blockDim.x;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int ix[2]; bool ok[2];
#pragma unroll
    for (int h = 0; h < 2; h++) { ix[h] = threadIdx.x + h * T; ok[h] = 4 * ix[h] < E; }
    auto load = [&](const float *p, int h) { return ok[h] ? __ldg(reinterpret_cast<const float4 *>(p) + ix[h]) : zero; };       /* weights: not an earlier kernel's work */
    const float *const wptr[6] = {a.post_ffw1, a.post_ffw2, a.post_ffw, a.ffn_norm, a.pre_ffw2, a.router_scale};
    float4 pre[6][2];
    if (FEW) {
#pragma unroll
        for (int k = FIN ? 0 : 3; k < (OUT ? 6 : 3); k++)
#pragma unroll
            for (int h = 0; h < 2; h++) pre[k][h] = load(wptr[k], h);
    }
    auto vec = [&](int k, int h) { return FEW ? pre[k][h] : load(wptr[k], h); };
    sp_pdl_wait();
    sp_pdl_next();
    if (OUT && t == 0) for (int k = threadIdx.x; k < d.NE; k += T) a.count[k] = 0;
    const size_t row = (size_t)t * E;
    auto row4 = [&](const float *p, int h) {
        if (!ok[h]) return zero;
        if (VEC) return __ldcs(reinterpret_cast<const float4 *>(p) + ix[h]);
        const float *q = p + 4 * ix[h];
        return make_float4(__ldcs(q), __ldcs(q + 1), __ldcs(q + 2), __ldcs(q + 3));
    };
    float4 x[2];
#pragma unroll
    for (int h = 0; h < 2; h++) x[h] = row4(a.x + row, h);
    if (FIN) {
        float4 dn[2], c[2] = {zero, zero};
#pragma unroll
        for (int h = 0; h < 2; h++) dn[h] = row4(a.dn + row, h);
#pragma unroll
        for (int k0 = 0; k0 < SP_MAX_NU; k0 += KB) {            /* KB pair rows in flight */
            float4 o[KB][2]; float cw[KB];
#pragma unroll
            for (int k = 0; k < KB; k++) {
                cw[k] = 0.0f; o[k][0] = o[k][1] = zero;
                if (k0 + k < NU) {
                    const size_t p = (size_t)t * NU + k0 + k;
                    cw[k] = a.cw[p];
                    const float *r = a.eo + (size_t)(a.pair_index ? a.pair_index[p] : (int)p) * E;
#pragma unroll
                    for (int h = 0; h < 2; h++) o[k][h] = row4(r, h);
                }
            }
#pragma unroll
            for (int k = 0; k < KB; k++)
                if (k0 + k < NU)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        c[h].x = __fadd_rn(c[h].x, __fmul_rn(cw[k], o[k][h].x)); c[h].y = __fadd_rn(c[h].y, __fmul_rn(cw[k], o[k][h].y));
                        c[h].z = __fadd_rn(c[h].z, __fmul_rn(cw[k], o[k][h].z)); c[h].w = __fadd_rn(c[h].w, __fmul_rn(cw[k], o[k][h].w));
                    }
        }
        double s2[2] = {sumsq4(dn[0]) + sumsq4(dn[1]), sumsq4(c[0]) + sumsq4(c[1])};
        block_sum<2>(s2, red[0]);
        const float sc1 = rms_scale_from(s2[0], E, d.eps), sc2 = rms_scale_from(s2[1], E, d.eps);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float4 m = scale4(dn[h], sc1, vec(0, h)), u = scale4(c[h], sc2, vec(1, h));
            dn[h] = make_float4(__fadd_rn(m.x, u.x), __fadd_rn(m.y, u.y), __fadd_rn(m.z, u.z), __fadd_rn(m.w, u.w));
        }
        double s1[1] = {sumsq4(dn[0]) + sumsq4(dn[1])};
        block_sum<1>(s1, red[1]);
        const float sc3 = rms_scale_from(s1[0], E, d.eps);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float4 r = scale4(dn[h], sc3, vec(2, h));
            x[h] = make_float4(__fadd_rn(x[h].x, r.x), __fadd_rn(x[h].y, r.y), __fadd_rn(x[h].z, r.z), __fadd_rn(x[h].w, r.w));
            if (ok[h]) {
                if (VEC) reinterpret_cast<float4 *>(a.y + row)[ix[h]] = x[h];
                else { float *q = a.y + row + 4 * ix[h]; q[0] = x[h].x; q[1] = x[h].y; q[2] = x[h].z; q[3] = x[h].w; }
            }
        }
    }
    if (OUT) {
        double s1[1] = {sumsq4(x[0]) + sumsq4(x[1])};
        block_sum<1>(s1, red[2]);
        const float sc = rms_scale_from(s1[0], E, d.eps);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = ix[h];
            const float4 n = scale4(x[h], sc, vec(3, h)), in = scale4(x[h], sc, vec(4, h));
            if (ok[h]) {
                const float4 xs = make_float4(__fmul_rn(x[h].x, sc), __fmul_rn(x[h].y, sc), __fmul_rn(x[h].z, sc), __fmul_rn(x[h].w, sc));
                reinterpret_cast<float4 *>(a.rin + row)[i] = scale4(xs, d.inv_sqrt_e, vec(5, h));
            }
            if (OUT == kOutInt8) {
                quant_quad(n, ok[h], i, a.nx_q + (size_t)t * sp_act_pitch(E), E);
                quant_quad(in, ok[h], i, a.in_q + (size_t)t * sp_act_pitch(E), E);
            } else if (OUT == kOutSplit) {
                split_quad(n, ok[h], i, a.nx_hi + row, a.nx_lo + row);
                split_quad(in, ok[h], i, a.in_hi + row, a.in_lo + row);
            } else if (ok[h]) {
                reinterpret_cast<float4 *>(a.nx_f + row)[i] = n;
                reinterpret_cast<float4 *>(a.in_f + row)[i] = in;
            }
            if (a.rows_f && ok[h]) reinterpret_cast<float4 *>(a.rows_f + row)[i] = in;
        }
    }
}
/* End of a layer + beginning of the next: as two kernels of 256 threads that walked the row in shared memory 229 us for 4096
 * tokens, as this one 111 us (625 MB of it pair rows and rows in and out). FEW while no SM has a second block: a layer of 65 /
 * 100 tokens 184 / 237 us with it and 193 / 245 without (decode arithmetic, E 2816; prefill 224 / 226 and 229 / 231), the
 * same within 1% from 148 to 444. */
template <bool FIN, int OUT>
cudaError_t launch_token(const SpDims &d, int M, const TokArgs &a, cudaStream_t st, int *nl) {
    const unsigned threads = (unsigned)((d.E / 8 + 31) & ~31);
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const bool wide = d.E > 3072, few = M <= sms;
    if (((uintptr_t)a.x | (uintptr_t)a.eo | (uintptr_t)a.y) & 15) {
        /* only the end of a layer meets a caller's pointers as they are (sp_moe_forward_dev, sp_moe_ep_finish_dev); an x that a
         * layer begins with is copied to the handle's own buffer first */
        if constexpr (FIN && OUT == kOutNone) return sp_launch(wide ? k_b_token<FIN, OUT, true, false, false> : k_b_token<FIN, OUT, false, false, false>, dim3((unsigned)M), threads, 0, st, nl, d, a);
        else return cudaErrorInvalidValue;
    }
    return sp_launch(wide ? (few ? k_b_token<FIN, OUT, true, true> : k_b_token<FIN, OUT, true, false>) : (few ? k_b_token<FIN, OUT, false, true> : k_b_token<FIN, OUT, false, false>),
                     dim3((unsigned)M), threads, 0, st, nl, d, a);
}
void set_prep(TokArgs &a, const SpLayerDev &L, const BView &v, SpTcPlan *split) {
    a.ffn_norm = L.ffn_norm; a.pre_ffw2 = L.pre_ffw2; a.router_scale = L.router_scale; a.rin = v.rin; a.count = v.count;
    a.nx_q = v.nx_q; a.in_q = v.in_q; a.nx_f = v.nx_f; a.in_f = v.in_f;
    if (split) sp_tc_inputs(split, &a.nx_hi, &a.nx_lo, &a.in_hi, &a.in_lo);
}
void set_finish(TokArgs &a, const SpLayerDev &L, const BView &v, const float *eo, const int *pair_index, float *y) {
    a.dn = v.dn; a.eo = eo; a.cw = v.cw; a.pair_index = pair_index; a.post_ffw1 = L.post_ffw1; a.post_ffw2 = L.post_ffw2; a.post_ffw = L.post_ffw; a.y = y;
}

/* ---------------------------------------------------------------- K2: router logits, fp32, fixed order
 * lane l takes the float4 groups q = l, l+32, ... with acc = fma(w, x, acc) over the four
 * elements in order, then the shuffle tree (the same order the decode kernel uses). One block =
 * 32 experts x 16 tokens; E is walked in chunks of 32 float4 groups staged in shared memory, and
 * each warp keeps an 8-expert x 8-token register tile (16 shared-memory loads per 256 FMAs), so every
 * (expert, token) chain keeps the order above while 64 independent chains hide the FMA latency. Bound by shared memory
 * (as many cycles of loads as of FMAs, and the copies in) and the last wave: 129 us at 4096 tokens with two stages and 64
 * separate trees, 90 us with four stages, one barrier a chunk and the trees together. */
constexpr int kRouterTE = 32, kRouterTT = 16;
constexpr int kRouterStages = 4;
constexpr size_t kRouterSmem = kRouterStages * (size_t)(kRouterTE + kRouterTT) * 32 * sizeof(float4);     /* stages of 24 KB */
/* 16-byte asynchronous copy that writes zeros when `take` is false (the source address stays valid either way) */
__device__ __forceinline__ void cp_async16_zfill(void *smem_dst, const void *src, bool take) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"((unsigned)__cvta_generic_to_shared(smem_dst)), "l"(src), "r"(take ? 16 : 0) : "memory");
}
__global__ void __launch_bounds__(256, 2) k_b_router(SpDims d, SpLayerDev L, BView v, int M) {
    extern __shared__ __align__(16) float4 rsm[];              /* [kRouterStages] x { w[32][32], x[16][32] }: the next chunks land while this one is used */
    const int E = d.E, G = E >> 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int we = warp & 3, wt = warp >> 2;
    const int e0 = blockIdx.x * kRouterTE, t0 = blockIdx.y * kRouterTT;
    sp_pdl_wait();
    sp_pdl_next();
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
    auto stage = [&](int c0, int buf) {                         /* warp w stages expert rows w, w+8, w+16, w+24 and token rows w, w+8 */
        float4 *wS = rsm + (size_t)buf * (kRouterTE + kRouterTT) * 32, *xS = wS + kRouterTE * 32;
        const int gg = c0 + lane; const bool gok = gg < G; const int gc = gok ? gg : 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int row = warp + 8 * k; const bool ok = gok && e0 + row < d.NE;
            cp_async16_zfill(wS + row * 32 + lane, reinterpret_cast<const float4 *>(L.router_w + (size_t)(ok ? e0 + row : 0) * E) + gc, ok);
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int row = warp + 8 * k; const bool ok = gok && t0 + row < M;
            cp_async16_zfill(xS + row * 32 + lane, reinterpret_cast<const float4 *>(v.rin + (size_t)(ok ? t0 + row : 0) * E) + gc, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int nch = (G + 31) >> 5;
    for (int c = 0; c < kRouterStages - 1; c++) { if (c < nch) stage(32 * c, c); else asm volatile("cp.async.commit_group;" ::: "memory"); }
    for (int c = 0, buf = 0, nbuf = kRouterStages - 1; c < nch; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRouterStages - 2) : "memory");
        __syncthreads();                                        /* chunk c is there; every warp has read chunk c - 1, whose place the new one takes */
        if (c + kRouterStages - 1 < nch) stage(32 * (c + kRouterStages - 1), nbuf); else asm volatile("cp.async.commit_group;" ::: "memory");
        const float4 *wS = rsm + (size_t)buf * (kRouterTE + kRouterTT) * 32, *xS = wS + kRouterTE * 32;
        buf = buf == kRouterStages - 1 ? 0 : buf + 1; nbuf = nbuf == kRouterStages - 1 ? 0 : nbuf + 1;
        float4 w[8];                                            /* zero padding beyond E leaves acc unchanged: fma(0, 0, acc) = acc */
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = wS[(8 * we + i) * 32 + lane];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float4 x = xS[(8 * wt + j) * 32 + lane];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float a = acc[i][j];
                a = __fmaf_rn(w[i].x, x.x, a); a = __fmaf_rn(w[i].y, x.y, a);
                a = __fmaf_rn(w[i].z, x.z, a); a = __fmaf_rn(w[i].w, x.w, a);
                acc[i][j] = a;
            }
        }
    }
    /* all 64 sums at once: at every level of the tree a lane keeps half of the values and hands the others over (the pairs that
     * warp_tree adds, 62 shuffles instead of 320); it ends with two neighbouring tokens of one expert */
    float f[64];
#pragma unroll
    for (int k = 0; k < 64; k++) f[k] = acc[k >> 3][k & 7];
#pragma unroll
    for (int o = 16, n = 32; o > 0; o >>= 1, n >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int k = 0; k < 32; k++)
            if (k < n) f[k] = (hi ? f[k + n] : f[k]) + __shfl_xor_sync(0xffffffffu, hi ? f[k] : f[k + n], o);
    }
    const int e = e0 + 8 * we + (lane >> 2), t = t0 + 8 * wt + 2 * (lane & 3);
    if (e < d.NE) {
        const float bias = L.router_bias ? __ldg(L.router_bias + e) : 0.0f;
#pragma unroll
        for (int j = 0; j < 2; j++)
            if (t + j < M) v.logits[(size_t)(t + j) * d.NE + e] = L.router_bias ? __fadd_rn(f[j], bias) : f[j];
    }
}

/* The same logits for a handful of tokens: one block per (expert, eight tokens), so that a small batch
 * still spreads over the machine (it is bound by the latency of one block's loop, not by arithmetic).
 * The expert's row is staged in shared memory; warp w takes token 8*blockIdx.y + w, lane l the float4
 * groups l, l+32, ... in the order given above. */
__global__ void __launch_bounds__(256) k_b_router_small(SpDims d, SpLayerDev L, BView v, int M) {
    extern __shared__ __align__(16) float4 rw[];               /* [E/4] */
    const int E = d.E, G = E >> 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = blockIdx.x;
    const float4 *wrow = reinterpret_cast<const float4 *>(L.router_w + (size_t)e * E);
    for (int g = threadIdx.x; g < G; g += 256) rw[g] = __ldg(wrow + g);      /* a weight: fetched before the wait */
    sp_pdl_wait();
    sp_pdl_next();
    __syncthreads();
    const int t = blockIdx.y * 8 + warp;
    if (t >= M) return;
    const float4 *x = reinterpret_cast<const float4 *>(v.rin + (size_t)t * E);
    float acc = 0.0f;
#pragma unroll 8
    for (int g = lane; g < G; g += 32) {
        const float4 w = rw[g], xv = x[g];
        acc = __fmaf_rn(w.x, xv.x, acc); acc = __fmaf_rn(w.y, xv.y, acc);
        acc = __fmaf_rn(w.z, xv.z, acc); acc = __fmaf_rn(w.w, xv.w, acc);
    }
    const float r = warp_tree(acc);
    if (lane == 0) v.logits[(size_t)t * d.NE + e] = L.router_bias ? __fadd_rn(r, __ldg(L.router_bias + e)) : r;
}
/* up to this many tokens the per-(expert, eight tokens) blocks beat the tiled kernel. A layer of E 2816 and 128 experts, small /
 * tiled: 38.8 / 51.4 us at 2 tokens, 91.6 / 103.7 at 16, 119.4 / 129.6 at 32, 173.6 / 179.9 at 64 (decode arithmetic); 223.0 /
 * 224.2 at 80, 226.1 / 226.2 at 96, 234.3 / 236.7 at 128, 253.1 / 246.7 at 160, 412 / 385 at 512 (prefill). */
constexpr int kRouterSmallM = 64;
cudaError_t launch_router(const SpDims &d, const SpLayerDev &L, BView &v, int M, cudaStream_t st, int *nl) {
    if (M <= kRouterSmallM && (size_t)d.E * 4 <= 48 * 1024)
        return sp_launch(k_b_router_small, dim3((unsigned)d.NE, (unsigned)((M + 7) / 8)), 256, (size_t)d.E * 4, st, nl, d, L, v, M);
    return sp_launch(k_b_router, dim3((d.NE + kRouterTE - 1) / kRouterTE, (M + kRouterTT - 1) / kRouterTT), 256, kRouterSmem, st, nl, d, L, v, M);
}

/* ---------------------------------------------------------------- K3: moe_topk_host (CF:6220-6240) + bucketing by expert (CF:8594-8624) */
struct TopkOut { int32_t *sel; float *wts; int *status; };
/* the selection of one token, expert e in place k of the descending order with probability p: clamped weights, ascending
 * slots, bucketing */
__device__ __forceinline__ void topk_store(const SpDims &d, const SpLayerDev &L, const BView &v, int M, int tok, int k, int e, float p, float wsum, int slot, const TopkOut &o) {
    if (wsum < 6.103515625e-5f) wsum = 6.103515625e-5f;
    const float w = __fdiv_rn(p, wsum);
    const int pair = tok * d.NU + slot;
    v.sel_asc[pair] = e;
    v.cw[pair] = __fmul_rn(w, __ldg(L.dexps_scale + e));                 /* CF:8709 */
    const int pos = atomicAdd(&v.count[e], 1);
    v.pairpos[pair] = pos;
    if (pos < M) v.list[(size_t)e * M + pos] = pair; else atomicExch(o.status, SP_KERR_OVERFLOW);
    if (o.sel) o.sel[(size_t)tok * d.NU + k] = e;
    if (o.wts) o.wts[(size_t)tok * d.NU + k] = w;
}
/* NE <= 128: one warp per token, four candidates a lane; NU rounds of (largest probability, then the lowest id among its
 * holders), the order moe_topk_host's strict > insertion produces. key = bits(p) + 1 for a usable probability (p >= 0, so
 * its bits order like its value), 0 for a NaN or an absent candidate. */
__global__ void __launch_bounds__(128) k_b_topk_warp(SpDims d, SpLayerDev L, BView v, int M, TopkOut o) {
    const int lane = threadIdx.x & 31, tok = blockIdx.x * 4 + (threadIdx.x >> 5), NE = d.NE, NU = d.NU;
    sp_pdl_wait();
    sp_pdl_next();
    if (tok >= M) return;
    const float *lg = v.logits + (size_t)tok * NE;
    float l[4], mx = -INFINITY; bool bad = false;
#pragma unroll
    for (int k = 0; k < 4; k++) { l[k] = lane + 32 * k < NE ? lg[lane + 32 * k] : -INFINITY; bad |= l[k] != l[k]; mx = fmaxf(mx, l[k]); }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, q));
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(o.status, SP_KERR_NAN_ROUTER);
    double ex[4], sum = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) { ex[k] = lane + 32 * k < NE ? exp((double)l[k] - (double)mx) : 0.0; sum += ex[k]; }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, q);
    unsigned key[4];
#pragma unroll
    for (int k = 0; k < 4; k++) { const float p = (float)(ex[k] / sum); key[k] = (lane + 32 * k < NE && p == p) ? __float_as_uint(p) + 1u : 0u; }
    int e = lane < NE ? lane : 0; float p = 0.0f;               /* lane r keeps the r-th of the descending order */
#pragma unroll 1
    for (int r = 0; r < NU; r++) {
        unsigned lm = key[0] > key[1] ? key[0] : key[1]; const unsigned l2 = key[2] > key[3] ? key[2] : key[3]; lm = lm > l2 ? lm : l2;
        const unsigned m = __reduce_max_sync(0xffffffffu, lm);
        if (m == 0u) break;
        unsigned cand = 0x7fffffffu;
#pragma unroll
        for (int k = 3; k >= 0; k--) if (key[k] == m) cand = (unsigned)(lane + 32 * k);
        const unsigned w = __reduce_min_sync(0xffffffffu, cand);
#pragma unroll
        for (int k = 0; k < 4; k++) if ((unsigned)(lane + 32 * k) == w) key[k] = 0u;
        if (lane == r) { e = (int)w; p = __uint_as_float(m - 1u); }
    }
    float wsum = 0.0f; int slot = 0;
    for (int k = 0; k < NU; k++) {
        wsum = __fadd_rn(wsum, __shfl_sync(0xffffffffu, p, k));
        slot += __shfl_sync(0xffffffffu, e, k) < e;
    }
    if (lane < NU) topk_store(d, L, v, M, tok, lane, e, p, wsum, slot, o);
}
/* any NE: one block per token, the rank of a candidate counted against all others */
__global__ void __launch_bounds__(256) k_b_topk(SpDims d, SpLayerDev L, BView v, int M, TopkOut o) {
    extern __shared__ __align__(16) unsigned char tsm[];
    const int NE = d.NE, NU = d.NU, t = threadIdx.x, tok = blockIdx.x;
    double *ex = reinterpret_cast<double *>(tsm);               /* [NE] */
    float *p = reinterpret_cast<float *>(ex + NE);              /* [NE] */
    __shared__ double red[8];
    __shared__ float wmax[8];
    __shared__ int sel_desc[SP_MAX_NU];
    __shared__ float p_desc[SP_MAX_NU];
    sp_pdl_wait();
    sp_pdl_next();
    const float *lg = v.logits + (size_t)tok * NE;
    float mx = -INFINITY; int bad = 0;
    for (int i = t; i < NE; i += 256) { const float l = lg[i]; if (l != l) bad = 1; mx = fmaxf(mx, l); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); bad |= __shfl_xor_sync(0xffffffffu, bad, o); }
    if ((t & 31) == 0) wmax[t >> 5] = mx;
    if (bad && (t & 31) == 0) atomicExch(o.status, SP_KERR_NAN_ROUTER);
    __syncthreads();
    mx = wmax[0];
#pragma unroll
    for (int w = 1; w < 8; w++) mx = fmaxf(mx, wmax[w]);
    double part = 0.0;
    for (int i = t; i < NE; i += 256) { const double e = exp((double)lg[i] - (double)mx); ex[i] = e; part += e; }
    part = warp_sum_f64(part);
    if ((t & 31) == 0) red[t >> 5] = part;
    __syncthreads();
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < 8; w++) sum += red[w];
    for (int i = t; i < NE; i += 256) p[i] = (float)(ex[i] / sum);
    if (t < SP_MAX_NU) { sel_desc[t] = t < NE ? t : 0; p_desc[t] = 0.0f; }
    __syncthreads();
    for (int i = t; i < NE; i += 256) {
        const float pi = p[i]; int r = 0;
        for (int j = 0; j < NE; j++) { const float pj = p[j]; r += (pj > pi) || (pj == pi && j < i); }
        if (r < NU && pi == pi) { sel_desc[r] = i; p_desc[r] = pi; }
    }
    __syncthreads();
    if (t < NU) {
        float wsum = 0.0f;
        for (int k = 0; k < NU; k++) wsum = __fadd_rn(wsum, p_desc[k]);
        const int e = sel_desc[t];
        int slot = 0;
        for (int j = 0; j < NU; j++) slot += (sel_desc[j] < e);
        topk_store(d, L, v, M, tok, t, e, p_desc[t], wsum, slot, o);
    }
}
cudaError_t launch_topk(const SpDims &d, const SpLayerDev &L, BView &v, int M, int32_t *sel, float *wts, int *status, cudaStream_t st, int *nl) {
    const TopkOut o{sel, wts, status};
    if (d.NE <= 128) return sp_launch(k_b_topk_warp, dim3((unsigned)((M + 3) / 4)), 128, 0, st, nl, d, L, v, M, o);
    return sp_launch(k_b_topk, dim3((unsigned)M), 256, (size_t)d.NE * 12, st, nl, d, L, v, M, o);
}

/* ---------------------------------------------------------------- per-row activation quant (CF:1725-1746): received rows of an expert-parallel run */
template <bool VEC>                                                             /* a caller's rows on some other float boundary: single floats */
__global__ void __launch_bounds__(1024) k_b_quant_rows(const float *x, int n, unsigned char *act) {
    const size_t r = blockIdx.x;
    const int i = threadIdx.x;
    const bool ok = 4 * i < n;
    sp_pdl_wait();
    sp_pdl_next();
    const float *p = x + r * n + 4 * i;
    const float4 f = !ok ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : VEC ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
    quant_quad(f, ok, i, act + r * sp_act_pitch(n), n);
}

/* ---------------------------------------------------------------- K4/K6, floating-point flavour without the tensor cores
 * (the integer flavour's rows are rows_mma.cu's). One warp per output row (or gate/up row pair); its codes and block scales are loaded ONCE into
 * registers and reused for every activation in the group's list, so each weight byte is read from
 * HBM once per layer however many tokens share the expert. grid.y = group (expert, or 0 for the
 * shared expert whose list is every token). */
struct GroupArgs {
    const uint8_t *codes; const uint16_t *bs;      /* tensor base */
    long long rows_per_group;                      /* row stride between groups */
    const int *count, *list; int list_stride;      /* per-group lists (NULL list = identity 0..M-1) */
    const int *offset;                             /* or: group g owns items [offset[g], offset[g+1]) (rows sorted by expert) */
    const int *index;                              /* with offset: sorted position -> row in the buffers (NULL = identity) */
    int M, in, rows;                               /* rows (or pairs) per group */
    int up_off;                                    /* PAIR: row offset of the up row */
    const uint8_t *ucodes; const uint16_t *ubs;    /* PAIR with a separate up tensor (shared expert), else NULL */
    int act_div;                                   /* activation row = item / act_div (NU for routed gate|up, 1 otherwise) */
    const int *act_index;                          /* with offset: sorted position -> activation row, when it is not the item's own row (NULL = item / act_div) */
    const float *xf;
    float *out; int out_stride;                    /* out[item * out_stride + row] */
};

template <int NIT>
__device__ __forceinline__ void load_row(const uint8_t *codes, const uint16_t *bs, int n32, int lane, int4 (&w)[NIT], float (&sc)[NIT]) {
#pragma unroll
    for (int i = 0; i < NIT; i++) {
        const int c = lane + 32 * i;
        if (c < n32) { w[i] = ld_stream16(codes + 16 * (size_t)c); sc[i] = h2f(ld_stream_u16(bs + c)); }
        else { w[i] = make_int4(0, 0, 0, 0); sc[i] = 0.0f; }
    }
}
/* flavour B: w = code * scale exactly (CF:1459-1463), fp32 dot */
template <int NIT>
__device__ __forceinline__ float dot_b(const int4 (&w)[NIT], const float (&sc)[NIT], int n32, int lane, const float *x) {
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < NIT; i++) {
        const int c = lane + 32 * i;
        if (c < n32) {
            const float4 *xv = reinterpret_cast<const float4 *>(x + 32 * c);
            const int words[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
            float blk = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 x0 = xv[2 * k], x1 = xv[2 * k + 1];
                const int wd = words[k];
                blk = __fmaf_rn((float)(((wd & 0xF) ^ 8) - 8), x0.x, blk);
                blk = __fmaf_rn((float)((((wd >> 4) & 0xF) ^ 8) - 8), x0.y, blk);
                blk = __fmaf_rn((float)((((wd >> 8) & 0xF) ^ 8) - 8), x0.z, blk);
                blk = __fmaf_rn((float)((((wd >> 12) & 0xF) ^ 8) - 8), x0.w, blk);
                blk = __fmaf_rn((float)((((wd >> 16) & 0xF) ^ 8) - 8), x1.x, blk);
                blk = __fmaf_rn((float)((((wd >> 20) & 0xF) ^ 8) - 8), x1.y, blk);
                blk = __fmaf_rn((float)((((wd >> 24) & 0xF) ^ 8) - 8), x1.z, blk);
                blk = __fmaf_rn((float)((((wd >> 28) & 0xF) ^ 8) - 8), x1.w, blk);
            }
            acc = __fmaf_rn(sc[i], blk, acc);
        }
    }
    return warp_tree(acc);
}

template <bool PAIR, int NIT>
__global__ void __launch_bounds__(256) k_b_rows(GroupArgs g) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = blockIdx.y;
    int first = 0, cnt;
    if (g.offset) {                      /* caller-supplied ranges: keep them inside the g.M rows that exist */
        int last = g.offset[grp + 1];
        first = g.offset[grp];
        first = first < 0 ? 0 : (first > g.M ? g.M : first);
        last = last > g.M ? g.M : last;
        cnt = last - first;
    } else cnt = g.count ? g.count[grp] : g.M;
    if (cnt <= 0) return;
    const int r = blockIdx.x * 8 + warp;
    if (r >= g.rows) return;
    const int n32 = g.in >> 5;
    const size_t rb = (size_t)g.in / 2;
    const size_t row = (size_t)grp * g.rows_per_group + r;
    int4 w0[NIT], w1[PAIR ? NIT : 1]; float s0[NIT], s1[PAIR ? NIT : 1];
    load_row<NIT>(g.codes + row * rb, g.bs + row * n32, n32, lane, w0, s0);
    if (PAIR) {
        if (g.ucodes) load_row<NIT>(g.ucodes + row * rb, g.ubs + row * n32, n32, lane, reinterpret_cast<int4(&)[NIT]>(w1), reinterpret_cast<float(&)[NIT]>(s1));
        else load_row<NIT>(g.codes + (row + g.up_off) * rb, g.bs + (row + g.up_off) * n32, n32, lane, reinterpret_cast<int4(&)[NIT]>(w1), reinterpret_cast<float(&)[NIT]>(s1));
    }
    const int *list = g.list ? g.list + (size_t)grp * g.list_stride : nullptr;
    for (int i = 0; i < cnt; i++) {
        const int item = list ? list[i] : (g.index ? g.index[first + i] : first + i);
        const size_t arow = (size_t)(g.act_index ? g.act_index[first + i] : item / g.act_div);
        const float *x = g.xf + arow * g.in;
        float o = dot_b<NIT>(w0, s0, n32, lane, x);
        if (PAIR) o = gelu_mul(o, dot_b<NIT>(reinterpret_cast<int4(&)[NIT]>(w1), reinterpret_cast<float(&)[NIT]>(s1), n32, lane, x));
        if (lane == 0) g.out[(size_t)item * g.out_stride + r] = o;
    }
}

template <bool PAIR>
void launch_rows(const GroupArgs &g, int groups, cudaStream_t st, int *nl) {
    const dim3 grid((unsigned)((g.rows + 7) / 8), (unsigned)groups);
    const int nit = ((g.in >> 5) + 31) >> 5;
    if (nit <= 1) k_b_rows<PAIR, 1><<<grid, 256, 0, st>>>(g);
    else if (nit == 2) k_b_rows<PAIR, 2><<<grid, 256, 0, st>>>(g);
    else if (nit == 3) k_b_rows<PAIR, 3><<<grid, 256, 0, st>>>(g);
    else k_b_rows<PAIR, 4><<<grid, 256, 0, st>>>(g);
    (*nl)++;
}

/* ---------------------------------------------------------------- K4/K6, integer flavour: the four row sets as segments of rows_mma.cu */
SpRowsSeg seg_shared_up(const SpDims &d, const SpLayerDev &L, int M, const BView &v) {
    SpRowsSeg s{};
    s.codes = L.sg_codes; s.bs = L.sg_bs; s.ucodes = L.su_codes; s.ubs = L.su_bs; s.in = d.E; s.rows = d.FFS; s.groups = 1; s.M = M; s.act_div = 1;
    s.act = v.nx_q; s.out_act = v.hd_q;
    return s;
}
SpRowsSeg seg_shared_down(const SpDims &d, const SpLayerDev &L, int M, const BView &v) {
    SpRowsSeg s{};
    s.codes = L.sd_codes; s.bs = L.sd_bs; s.in = d.FFS; s.rows = d.E; s.groups = 1; s.M = M; s.act_div = 1;
    s.act = v.hd_q; s.out_f = v.dn; s.out_stride = d.E;
    return s;
}
SpRowsSeg seg_routed_up(const SpDims &d, const SpLayerDev &L, int M, const unsigned char *act, const BView &v) {
    SpRowsSeg s{};
    s.codes = s.ucodes = L.gu_codes; s.bs = s.ubs = L.gu_bs; s.rows_per_group = 2LL * d.FFE; s.up_off = d.FFE; s.in = d.E; s.rows = d.FFE; s.groups = d.NE;
    s.M = M; s.act_div = 1; s.act = act; s.out_act = v.h_q;
    return s;
}
SpRowsSeg seg_routed_down(const SpDims &d, const SpLayerDev &L, int M, const BView &v, float *out) {
    SpRowsSeg s{};
    s.codes = L.dn_codes; s.bs = L.dn_bs; s.rows_per_group = d.E; s.in = d.FFE; s.rows = d.E; s.groups = d.NE; s.M = M; s.act_div = 1;
    s.act = v.h_q; s.out_f = out; s.out_stride = d.E;
    return s;
}

/* the experts of one layer: the inputs the prep half left -> dn and eo */
template <bool FA>
cudaError_t run_experts(const SpDims &d, const SpLayerDev &L, int M, BView &v, SpTcPlan *tc, int *status, cudaStream_t st, int *nl) {
    const int E = d.E, NE = d.NE, NU = d.NU, FFE = d.FFE, FFS = d.FFS;
    if (!FA && tc) return sp_tc_layer(tc, d, L, M, v.sel_asc, v.count, v.pairpos, v.dn, v.eo, status, st, nl);      /* prefill arithmetic on the tensor cores */
    if (FA) {
        /* gate|up of the shared and the routed experts, quantised as it leaves (CF:8348-8356, 8733-8737, 8958-8959), then down (CF:8358, 8739-8742, 8961) */
        SpRowsSeg up[2] = {seg_shared_up(d, L, M, v), seg_routed_up(d, L, M, v.in_q, v)};
        up[1].count = v.count; up[1].list = v.list; up[1].list_stride = M; up[1].act_div = NU;
        const cudaError_t e = sp_rows_launch(up, 2, true, (long long)M * NU, status, st, nl);
        if (e != cudaSuccess) return e;
        SpRowsSeg down[2] = {seg_shared_down(d, L, M, v), seg_routed_down(d, L, M, v, v.eo)};
        down[1].count = v.count; down[1].list = v.list; down[1].list_stride = M;
        return sp_rows_launch(down, 2, false, (long long)M * NU, status, st, nl);
    }
    GroupArgs g{};
    g.M = M;
    /* shared expert gate/up -> hd (CF:8348-8356) */
    g.codes = L.sg_codes; g.bs = L.sg_bs; g.ucodes = L.su_codes; g.ubs = L.su_bs; g.rows_per_group = 0; g.count = nullptr; g.list = nullptr;
    g.in = E; g.rows = FFS; g.up_off = 0; g.act_div = 1; g.xf = v.nx_f; g.out = v.hd; g.out_stride = FFS;
    launch_rows<true>(g, 1, st, nl);
    /* routed gate|up -> h (CF:8733-8737, 8958-8959) */
    g.codes = L.gu_codes; g.bs = L.gu_bs; g.ucodes = nullptr; g.ubs = nullptr; g.rows_per_group = 2LL * FFE; g.count = v.count; g.list = v.list; g.list_stride = M;
    g.in = E; g.rows = FFE; g.up_off = FFE; g.act_div = NU; g.xf = v.in_f; g.out = v.h; g.out_stride = FFE;
    launch_rows<true>(g, NE, st, nl);
    /* shared down -> dn (CF:8358) */
    g.codes = L.sd_codes; g.bs = L.sd_bs; g.rows_per_group = 0; g.count = nullptr; g.list = nullptr;
    g.in = FFS; g.rows = E; g.act_div = 1; g.xf = v.hd; g.out = v.dn; g.out_stride = E;
    launch_rows<false>(g, 1, st, nl);
    /* routed down -> eo (CF:8739-8742, 8961) */
    g.codes = L.dn_codes; g.bs = L.dn_bs; g.rows_per_group = E; g.count = v.count; g.list = v.list; g.list_stride = M;
    g.in = FFE; g.rows = E; g.act_div = 1; g.xf = v.h; g.out = v.eo; g.out_stride = E;
    launch_rows<false>(g, NE, st, nl);
    return cudaGetLastError();
}
template <bool FA>
cudaError_t run_layers(const SpDims &d, const SpLayerDev *layers, int n, int M, const float *x, float *y, int32_t *sel, float *wts,
                       BView &v, SpTcPlan *tc, int *status, cudaStream_t st, int *nl) {
    /* where the experts' kernels take int8 or split rows, the end of a layer and the beginning of the next are one launch */
    const bool split = !FA && tc, fused = FA || split;
    const float *cur = x;
    cudaError_t e = cudaSuccess;
    for (int li = 0; li < n && e == cudaSuccess; li++) {
        const SpLayerDev &L = layers[li];
        float *dst = li == n - 1 ? y : (li & 1) ? v.xb : v.xa;
        TokArgs a{};
        a.x = cur;
        if (li == 0 || !fused) {
            set_prep(a, L, v, split ? tc : nullptr);
            e = FA ? launch_token<false, kOutInt8>(d, M, a, st, nl) : split ? launch_token<false, kOutSplit>(d, M, a, st, nl)
                   : launch_token<false, kOutF32>(d, M, a, st, nl);
        }
        if (e == cudaSuccess) e = launch_router(d, L, v, M, st, nl);
        if (e == cudaSuccess) e = launch_topk(d, L, v, M, sel ? sel + (size_t)li * M * d.NU : nullptr, wts ? wts + (size_t)li * M * d.NU : nullptr, status, st, nl);
        if (e == cudaSuccess) e = run_experts<FA>(d, L, M, v, tc, status, st, nl);
        if (e != cudaSuccess) break;
        set_finish(a, L, v, v.eo, nullptr, dst);
        if (fused && li + 1 < n) {
            set_prep(a, layers[li + 1], v, split ? tc : nullptr);
            e = FA ? launch_token<true, kOutInt8>(d, M, a, st, nl) : launch_token<true, kOutSplit>(d, M, a, st, nl);
        } else e = launch_token<true, kOutNone>(d, M, a, st, nl);
        cur = dst;
    }
    return e;
}

/* per-expert counts -> exclusive offsets (NE is at most 1024: one block) */
__global__ void __launch_bounds__(1024) k_b_scan(const int *count, int n, int *off) {
    __shared__ int sh[1024];
    const int t = threadIdx.x;
    sh[t] = t < n ? count[t] : 0;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) { const int v = t >= d ? sh[t - d] : 0; __syncthreads(); sh[t] += v; __syncthreads(); }
    if (t < n) off[t + 1] = sh[t];
    if (t == 0) off[0] = 0;
}
/* one block per (token, expert) pair: its input row goes to position off[e] + pairpos of the send buffer.
 * With a capacity (rows per destination rank, experts owned in blocks of epr) the buffer is padded: the rows
 * for rank r start at r * capacity, so the exchange needs no split sizes; a block that would not fit is
 * reported through the error word. */
__global__ void __launch_bounds__(256) k_b_dispatch_rows(const float *in_f, const int *sel_asc, const int *pairpos, const int *off, int NU, int E,
                                                         int epr, int capacity, float *rows, int *pair_index, int *status) {
    const int p = blockIdx.x;
    const int e = sel_asc[p];
    int pos = off[e] + pairpos[p];
    if (capacity > 0) {
        const int owner = e / epr, in_block = pos - off[owner * epr];
        if (in_block >= capacity) {
            if (threadIdx.x == 0) { pair_index[p] = owner * capacity; atomicExch(status, SP_KERR_OVERFLOW); }
            return;
        }
        pos = owner * capacity + in_block;
    }
    if (threadIdx.x == 0) pair_index[p] = pos;
    if (!rows) return;                           /* positions only: the caller sends token rows instead of pair rows */
    const float4 *src = reinterpret_cast<const float4 *>(in_f + (size_t)(p / NU) * E);
    float4 *dst = reinterpret_cast<float4 *>(rows + (size_t)pos * E);
    for (int i = threadIdx.x; i < E / 4; i += 256) dst[i] = src[i];
}
/* ---- token dispatch: a token's input row goes to a destination rank once, however many of its NU experts live
 * there. Per destination r: the tokens with at least one expert on r, in token order (slot = rank among them), up to
 * cap_tokens rows; per pair (at its position in the padded pair order, pair_index) the slot of its token. The receiver
 * multiplies row  source * cap_tokens + slot  for the pair. */
__global__ void __launch_bounds__(1024) k_b_tok_scan(const int *sel_asc, int M, int NU, int epr, int n_ranks, int cap_tokens, int *slot, int *status) {
    __shared__ int wsum[32];
    __shared__ int carry;
    const int r = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < M; base += 1024) {
        const int tok = base + t;
        int flag = 0;
        if (tok < M) for (int k = 0; k < NU; k++) flag |= (sel_asc[tok * NU + k] / epr == r);
        const unsigned bal = __ballot_sync(0xffffffffu, flag);
        const int within = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) wsum[warp] = __popc(bal);
        __syncthreads();
        int before = carry;
        for (int w = 0; w < warp; w++) before += wsum[w];
        if (tok < M) {
            const int sl = before + within;
            slot[tok * n_ranks + r] = flag ? sl : -1;
            if (flag && sl >= cap_tokens) atomicExch(status, SP_KERR_OVERFLOW);
        }
        __syncthreads();
        if (t == 0) { int tot = 0; for (int w = 0; w < 32; w++) tot += wsum[w]; carry += tot; }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(256) k_b_tok_rows(const float *in_f, const int *slot, int n_ranks, int cap_tokens, int E, float *tokrows) {
    const int tok = blockIdx.x, r = blockIdx.y;
    const int sl = slot[tok * n_ranks + r];
    if (sl < 0 || sl >= cap_tokens) return;
    const float4 *src = reinterpret_cast<const float4 *>(in_f + (size_t)tok * E);
    float4 *dst = reinterpret_cast<float4 *>(tokrows + ((size_t)r * cap_tokens + sl) * E);
    for (int i = threadIdx.x; i < E / 4; i += 256) dst[i] = src[i];
}
__global__ void __launch_bounds__(256) k_b_tok_idx(const int *sel_asc, const int *pair_index, const int *slot, int np, int NU, int epr, int n_ranks, int cap_tokens, int *tokidx) {
    const int p = blockIdx.x * 256 + threadIdx.x;
    if (p >= np) return;
    const int r = sel_asc[p] / epr;
    int sl = slot[(p / NU) * n_ranks + r];
    sl = sl < 0 ? 0 : (sl >= cap_tokens ? cap_tokens - 1 : sl);
    tokidx[pair_index[p]] = sl;
}
/* receiver: sorted position p -> the row of the pair's token among the token rows that arrived */
__global__ void __launch_bounds__(256) k_b_in_index(const int *row_index, const int *tokidx_recv, int n, int capacity, int cap_tokens, int n_ranks, int *in_index) {
    const int p = blockIdx.x * 256 + threadIdx.x;
    if (p >= n) return;
    const int a = row_index[p];                              /* arrival slot of the pair: source * capacity + position in the source's block */
    const int src = a / capacity;
    int sl = tokidx_recv[a];
    sl = sl < 0 ? 0 : (sl >= cap_tokens ? cap_tokens - 1 : sl);
    in_index[p] = (src < n_ranks ? src : n_ranks - 1) * cap_tokens + sl;
}
/* what a rank received through the padded exchange: source s's block starts at row s * capacity and holds
 * its rows for this rank's experts, sorted by expert. counts_all[s][e] = pairs of expert e on rank s.
 * Writes offsets[NE+1] (sorted position range of every expert; empty outside this rank's experts) and
 * row_index[n_ranks * capacity] (sorted position -> arrival row; 0 beyond the rows that exist). */
__global__ void __launch_bounds__(256) k_b_recv_layout(const int *counts_all, int NE, int n_ranks, int rank, int capacity, int *offsets, int *row_index) {
    extern __shared__ int lsm[];                 /* cnt[nb], sorted_start[nb + 1], arrival_start[nb], all in (expert, source) order */
    const int epr = NE / n_ranks, nb = epr * n_ranks, e0 = rank * epr;
    int *cnt = lsm, *sorted_start = lsm + nb, *arrival_start = lsm + 2 * nb + 1;
    for (int b = threadIdx.x; b < nb; b += 256) cnt[b] = counts_all[(b % n_ranks) * NE + e0 + b / n_ranks];
    __syncthreads();
    /* A source whose block for this rank overflowed kept only its first `capacity` rows, in expert order
     * (k_b_dispatch_rows drops the rest and sets the error word) but still reports its full counts: clamp
     * each source's running total to the capacity, so every index below stays inside the receive buffer. */
    for (int s_ = threadIdx.x; s_ < n_ranks; s_ += 256) {
        int a = 0;
        for (int e = 0; e < epr; e++) {
            int c = cnt[e * n_ranks + s_];
            c = c < 0 ? 0 : c;
            if (c > capacity - a) c = capacity - a;
            cnt[e * n_ranks + s_] = c;
            arrival_start[e * n_ranks + s_] = s_ * capacity + a;
            a += c;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int b = 0; b < nb; b++) { sorted_start[b] = acc; acc += cnt[b]; }
        sorted_start[nb] = acc;
    }
    __syncthreads();
    const int total = sorted_start[nb];
    for (int e = threadIdx.x; e <= NE; e += 256)
        offsets[e] = e < e0 ? 0 : (e >= e0 + epr ? total : sorted_start[(e - e0) * n_ranks]);
    for (int p = threadIdx.x; p < n_ranks * capacity; p += 256) {
        int v = 0;
        if (p < total) {
            int lo = 0, hi = nb - 1;               /* the block that holds sorted position p */
            while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (sorted_start[mid] <= p) lo = mid; else hi = mid - 1; }
            v = arrival_start[lo] + (p - sorted_start[lo]);
        }
        row_index[p] = v;
    }
}

/* ---------------------------------------------------------------- expert-parallel stages
 * The layer cut at the two places where (token, expert) pairs change GPU:
 *   route   : norms, router, top-k, the shared expert (kept in this handle's scratch), and the
 *             routed experts' input rows;
 *   experts : gate|up GeGLU + down for rows that arrive sorted by expert, on whichever GPU owns
 *             those experts (any subset: empty groups cost nothing);
 *   finish  : ordered combine of the returned pair rows + the recombine.
 * The arithmetic of each pair is the single-GPU batched path's, so a split run is bit-identical. */
/* the shared (always-on) expert of the tokens the last route call prepared: nx -> dn in the scratch */
/* phase 0 = the whole shared expert; 1 = gate/up + GeGLU only (hd stays in the scratch); 2 = the down rows only */
template <bool FA>
cudaError_t ep_shared(const SpDims &d, const SpLayerDev &L, int M, BView &v, SpTcPlan *tc, int *status, cudaStream_t st, int *nl, int phase) {
    const int E = d.E, FFS = d.FFS;
    if (!FA && tc) return sp_tc_shared_expert(tc, d, L, M, v.nx_f, v.dn, status, st, nl, phase);
    if (FA) {
        const SpRowsSeg up = seg_shared_up(d, L, M, v), down = seg_shared_down(d, L, M, v);
        cudaError_t e = phase != 2 ? sp_rows_launch(&up, 1, true, M, status, st, nl) : cudaSuccess;
        if (e == cudaSuccess && phase != 1) e = sp_rows_launch(&down, 1, false, M, status, st, nl);
        return e;
    }
    GroupArgs g{};
    g.M = M; g.act_div = 1;
    if (phase != 2) {
        g.codes = L.sg_codes; g.bs = L.sg_bs; g.ucodes = L.su_codes; g.ubs = L.su_bs;
        g.in = E; g.rows = FFS; g.xf = v.nx_f; g.out = v.hd; g.out_stride = FFS;
        launch_rows<true>(g, 1, st, nl);
    }
    if (phase != 1) {
        g.codes = L.sd_codes; g.bs = L.sd_bs; g.ucodes = nullptr; g.ubs = nullptr;
        g.in = FFS; g.rows = E; g.xf = v.hd; g.out = v.dn; g.out_stride = E;
        launch_rows<false>(g, 1, st, nl);
    }
    return cudaGetLastError();
}

template <bool FA>
cudaError_t ep_route(const SpDims &d, const SpLayerDev &L, int M, const float *x, int32_t *sel_asc, float *cw, float *rows, int32_t *counts,
                     int32_t *pair_index, int32_t *sel, float *wts, int defer_shared, int n_ranks, int capacity, BView &v, SpTcPlan *tc, int *status,
                     cudaStream_t st, int *nl) {
    const int E = d.E, NE = d.NE, NU = d.NU;
    TokArgs a{};
    a.x = x;
    set_prep(a, L, v, nullptr);
    if (FA) a.rows_f = v.in_f;                                  /* the routed experts' input as fp32 rows too, for the dispatch */
    cudaError_t e = FA ? launch_token<false, kOutInt8>(d, M, a, st, nl)
                       : launch_token<false, kOutF32>(d, M, a, st, nl);
    if (e == cudaSuccess) e = launch_router(d, L, v, M, st, nl);
    if (e == cudaSuccess) e = launch_topk(d, L, v, M, sel, wts, status, st, nl);
    if (e != cudaSuccess) return e;
    /* the send buffer: rows sorted by expert (so also by owner), ready for the all-to-all */
    k_b_scan<<<1, 1024, 0, st>>>(v.count, NE, v.ep_off); (*nl)++;
    k_b_dispatch_rows<<<M * NU, 256, 0, st>>>(v.in_f, v.sel_asc, v.pairpos, v.ep_off, NU, E, capacity > 0 ? NE / n_ranks : NE, capacity, rows, pair_index, status); (*nl)++;
    e = cudaMemcpyAsync(counts, v.count, (size_t)4 * NE, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(sel_asc, v.sel_asc, (size_t)4 * M * NU, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(cw, v.cw, (size_t)4 * M * NU, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    if (defer_shared) return cudaGetLastError();
    return ep_shared<FA>(d, L, M, v, tc, status, st, nl, 0);
}

/* in_index (optional, with n_in input rows): sorted position -> input row, when several pairs share one input row
 * (token dispatch); the outputs still go to the pair's own row (row_index). */
template <bool FA>
cudaError_t ep_experts(const SpDims &d, const SpLayerDev &L, int R, const float *rows_in, const int32_t *row_index, const int32_t *offsets, float *rows_out,
                       const int32_t *in_index, int n_in, int owners, BView &v, SpTcPlan *tc, int *status, cudaStream_t st, int *nl) {
    const int E = d.E, NE = d.NE, FFE = d.FFE;
    if (R == 0) return cudaSuccess;
    if (!FA && tc) return sp_tc_routed(tc, d, L, R, owners, rows_in, in_index ? in_index : row_index, offsets, row_index, rows_out, status, st, nl);
    if (FA) {
        cudaError_t e = sp_launch((uintptr_t)rows_in & 15 ? k_b_quant_rows<false> : k_b_quant_rows<true>, dim3((unsigned)(in_index ? n_in : R)), (unsigned)((E / 4 + 31) & ~31), 0, st, nl, rows_in, E, v.ep_q);
        if (e != cudaSuccess) return e;
        SpRowsSeg up = seg_routed_up(d, L, R, v.ep_q, v), down = seg_routed_down(d, L, R, v, rows_out);
        up.offset = down.offset = offsets; up.index = down.index = row_index; up.act_index = in_index;      /* h has one row per pair */
        up.owners = down.owners = owners;
        e = sp_rows_launch(&up, 1, true, R, status, st, nl);
        return e != cudaSuccess ? e : sp_rows_launch(&down, 1, false, R, status, st, nl);
    }
    GroupArgs g{};
    g.M = R; g.offset = offsets; g.index = row_index; g.act_index = in_index;
    g.codes = L.gu_codes; g.bs = L.gu_bs; g.rows_per_group = 2LL * FFE;
    g.in = E; g.rows = FFE; g.up_off = FFE; g.act_div = 1; g.xf = rows_in; g.out = v.h; g.out_stride = FFE;
    launch_rows<true>(g, NE, st, nl);
    g.codes = L.dn_codes; g.bs = L.dn_bs; g.rows_per_group = E; g.act_index = nullptr;          /* h has one row per pair */
    g.in = FFE; g.rows = E; g.xf = v.h; g.out = rows_out; g.out_stride = E;
    launch_rows<false>(g, NE, st, nl);
    return cudaGetLastError();
}

}  // namespace

cudaError_t sp_batched_ep_route(const SpDims &d, const SpLayerDev &L, int flavour, int M, const float *x, int32_t *sel_asc, float *cw,
                                float *rows, int32_t *counts, int32_t *pair_index, int32_t *sel, float *wts, int defer_shared, int n_ranks, int capacity,
                                SpBatchedScratch *s, int *status, cudaStream_t st, int *nlaunch, int t0, int slice) {
    *nlaunch = 0;
    if (!s->base || t0 < 0 || t0 + M > s->max_tokens || slice < 0 || slice >= kSlices) return cudaErrorInvalidValue;
    BView v = bview_slice(d, s, t0, slice);
    return flavour == SP_MOE_FLAVOUR_DECODE ? ep_route<true>(d, L, M, x, sel_asc, cw, rows, counts, pair_index, sel, wts, defer_shared, n_ranks, capacity, v, s->tc, status, st, nlaunch)
                                            : ep_route<false>(d, L, M, x, sel_asc, cw, rows, counts, pair_index, sel, wts, defer_shared, n_ranks, capacity, v, s->tc, status, st, nlaunch);
}
cudaError_t sp_batched_ep_recv_layout(const SpDims &d, const int32_t *counts_all, int n_ranks, int rank, int capacity, int32_t *offsets, int32_t *row_index,
                                      cudaStream_t st, int *nlaunch) {
    *nlaunch = 1;
    const int nb = d.NE;                                    /* epr * n_ranks */
    k_b_recv_layout<<<1, 256, (size_t)(3 * nb + 1) * sizeof(int), st>>>(counts_all, d.NE, n_ranks, rank, capacity, offsets, row_index);
    return cudaGetLastError();
}
cudaError_t sp_batched_ep_shared(const SpDims &d, const SpLayerDev &L, int flavour, int M, SpBatchedScratch *s, int *status, cudaStream_t st, int *nlaunch, int t0, int slice, int phase) {
    *nlaunch = 0;
    if (!s->base || t0 < 0 || t0 + M > s->max_tokens || slice < 0 || slice >= kSlices || phase < 0 || phase > 2) return cudaErrorInvalidValue;
    BView v = bview_slice(d, s, t0, slice);
    return flavour == SP_MOE_FLAVOUR_DECODE ? ep_shared<true>(d, L, M, v, s->tc, status, st, nlaunch, phase) : ep_shared<false>(d, L, M, v, s->tc, status, st, nlaunch, phase);
}
cudaError_t sp_batched_ep_experts(const SpDims &d, const SpLayerDev &L, int flavour, int R, const float *rows_in, const int32_t *row_index, const int32_t *offsets,
                                  float *rows_out, SpBatchedScratch *s, int *status, cudaStream_t st, int *nlaunch, const int32_t *in_index, int n_in, int owners) {
    *nlaunch = 0;
    if (!s->base || R > s->max_rows || (in_index && (n_in <= 0 || n_in > s->max_rows))) return cudaErrorInvalidValue;
    BView v = bview(d, s);
    return flavour == SP_MOE_FLAVOUR_DECODE ? ep_experts<true>(d, L, R, rows_in, row_index, offsets, rows_out, in_index, n_in, owners, v, s->tc, status, st, nlaunch)
                                            : ep_experts<false>(d, L, R, rows_in, row_index, offsets, rows_out, in_index, n_in, owners, v, s->tc, status, st, nlaunch);
}
/* token dispatch, sender side (after sp_batched_ep_route of the same tokens with rows == NULL): tokrows
 * [n_ranks][cap_tokens][E], tokidx [n_ranks][capacity] (the pair order of the padded exchange), slot = scratch of
 * M * n_ranks ints */
cudaError_t sp_batched_ep_tokens(const SpDims &d, int M, int n_ranks, int capacity, int cap_tokens, const int32_t *sel_asc, const int32_t *pair_index,
                                 float *tokrows, int32_t *tokidx, int32_t *slot, SpBatchedScratch *s, int *status, cudaStream_t st, int *nlaunch, int t0, int slice) {
    *nlaunch = 0;
    if (!s->base || t0 < 0 || t0 + M > s->max_tokens || slice < 0 || slice >= kSlices || n_ranks <= 0 || d.NE % n_ranks || capacity <= 0 || cap_tokens <= 0) return cudaErrorInvalidValue;
    BView v = bview_slice(d, s, t0, slice);
    const int epr = d.NE / n_ranks;
    k_b_tok_scan<<<n_ranks, 1024, 0, st>>>(sel_asc, M, d.NU, epr, n_ranks, cap_tokens, slot, status); (*nlaunch)++;
    k_b_tok_rows<<<dim3((unsigned)M, (unsigned)n_ranks), 256, 0, st>>>(v.in_f, slot, n_ranks, cap_tokens, d.E, tokrows); (*nlaunch)++;
    k_b_tok_idx<<<(M * d.NU + 255) / 256, 256, 0, st>>>(sel_asc, pair_index, slot, M * d.NU, d.NU, epr, n_ranks, cap_tokens, tokidx); (*nlaunch)++;
    return cudaGetLastError();
}
/* token dispatch, receiver side (after sp_batched_ep_recv_layout): in_index[n_ranks * capacity] */
cudaError_t sp_batched_ep_in_index(const int32_t *row_index, const int32_t *tokidx_recv, int n_ranks, int capacity, int cap_tokens, int32_t *in_index,
                                   cudaStream_t st, int *nlaunch) {
    *nlaunch = 1;
    const int n = n_ranks * capacity;
    k_b_in_index<<<(n + 255) / 256, 256, 0, st>>>(row_index, tokidx_recv, n, capacity, cap_tokens, n_ranks, in_index);
    return cudaGetLastError();
}
cudaError_t sp_batched_ep_finish(const SpDims &d, const SpLayerDev &L, int M, const float *x, const float *pair_rows, const int32_t *pair_index, float *y,
                                 SpBatchedScratch *s, cudaStream_t st, int *nlaunch, int t0, int slice) {
    *nlaunch = 0;
    if (!s->base || t0 < 0 || t0 + M > s->max_tokens || slice < 0 || slice >= kSlices) return cudaErrorInvalidValue;
    BView v = bview_slice(d, s, t0, slice);
    TokArgs a{};
    a.x = x;
    set_finish(a, L, v, pair_rows, pair_index, y);
    return launch_token<true, kOutNone>(d, M, a, st, nlaunch);
}

cudaError_t sp_batched_alloc(const SpDims &d, int max_tokens, int max_rows, SpBatchedScratch *s, size_t *bytes) {
    s->base = nullptr; s->bytes = 0; s->max_tokens = max_tokens; *bytes = 0;
    s->max_rows = max_rows > max_tokens * d.NU ? max_rows : max_tokens * d.NU;
    s->bytes = blayout(d, max_tokens, s->max_rows, [](int, size_t) {});
    s->tc = nullptr;
    cudaError_t e = sp_rows_prepare();
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_b_router, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRouterSmem);
    if (e != cudaSuccess) return e;
    e = cudaMalloc(&s->base, s->bytes);
    if (e != cudaSuccess) { s->base = nullptr; return e; }
    *bytes = s->bytes;
    /* house convention: behaviour switches are SP_* variables read once. "simt" keeps prefill on the fp32 CUDA-core kernels. */
    const char *ev = getenv("SP_MOE_PREFILL_IMPL");
    if (max_tokens > 1 && sp_tc_supported(d) && !(ev && ev[0] == 's')) {
        size_t tb = 0;
        e = sp_tc_create(d, max_tokens, s->max_rows, &s->tc, &tb);
        if (e != cudaSuccess) { cudaFree(s->base); s->base = nullptr; return e; }
        *bytes += tb;
    }
    return cudaSuccess;
}
void sp_batched_free(SpBatchedScratch *s) {
    if (!s) return;
    if (s->tc) { sp_tc_destroy(s->tc); s->tc = nullptr; }
    if (s->base) cudaFree(s->base);
    s->base = nullptr;
}

cudaError_t sp_batched_forward(const SpDims &d, const SpLayerDev *layers_host, int lf, int nl_, int flavour, int M,
                               const float *x, float *y, int32_t *sel, float *wts,
                               SpBatchedScratch *s, int *status, cudaStream_t st, int *nlaunch) {
    *nlaunch = 0;
    if (!s->base || M > s->max_tokens) return cudaErrorInvalidValue;
    BView v = bview(d, s);
    return flavour == SP_MOE_FLAVOUR_DECODE ? run_layers<true>(d, layers_host + lf, nl_, M, x, y, sel, wts, v, s->tc, status, st, nlaunch)
                                            : run_layers<false>(d, layers_host + lf, nl_, M, x, y, sel, wts, v, s->tc, status, st, nlaunch);
}
