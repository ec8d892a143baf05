/* ext_hook.cu — the reference's MoE plugin hook for SwiGLU models with separate gate / up / down
 * expert tensors (its qwen36 service: sp_q36gpu_upload_experts / sp_q36gpu_moe,
 * src/backends/cuda/cuda_forward.cu:16203-16289, registered through q36_boot_moe_ext,
 * CF:16444-16454): a layer's experts are uploaded once under a tag; a call names the tag, the
 * expert ids and weights the HOST router chose, and a host x[E]; the result is
 *     y = sum_k wt[k] * Wd[idx[k]] . ( silu(Wg[idx[k]] . x) * (Wu[idx[k]] . x) )
 * accumulated in the caller's k order (dg_k_axpy, fused multiply-add), every matmul in the decode
 * arithmetic (gemv_w_packed: int8 per-16 activation quant + Q4B x int8 GEMV, CF:13566-13599).
 * Contract of the hook: 0 = handled (y filled), nonzero = not mine (unknown tag or other shape).
 * Where the reference enqueues NU x (gate, up, silu*mul, down, axpy) between two copies, a call here is
 * three launches and one synchronisation: x is read from page-locked memory and quantised; gate and up
 * rows of all chosen experts with silu*mul; down rows of all of them with the accumulation, written
 * to page-locked memory. What bounds a call (14 MB of weights at E 2048, FF 512, eight experts: 2 us of
 * HBM) is the latency of these steps: 8 us to enqueue, then 18.5 us of waiting (the kernels take 4, 7 and 12 us one by one, cold),
 * of 33 us with a ctypes caller. Eight calls in a row: 263 us, 1784 us with six launches per expert and
 * pageable copies. Only Q4B tensors are served here.
 */
#include "common.cuh"
#include "launch.cuh"
#include "../../include/sp_engine/moe_backend.h"
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

namespace {

constexpr int kExtT = 512, kExtW = kExtT / 32, kExtSlots = 16;     /* threads and warps of a CTA; experts per round of launches */

struct ExtPick { int idx[kExtSlots]; float wt[kExtSlots]; int n; };

/* 16 floats -> one int8 block (k_quant_act_int8, CF:1564-1585) in the layout q4b_chunk_dot expects */
__device__ __forceinline__ void ext_quant(const float *p, int4 *q, float *sx, int *corr) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 4; i++) { const float4 f = reinterpret_cast<const float4 *>(p)[i]; v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w; }
    quant_block16_store(v, q, sx, corr);
}
__global__ void __launch_bounds__(256) k_ext_quant(const float *x, int E, int4 *q, float *sx, int *corr) {
    sp_pdl_wait();
    sp_pdl_next();
    for (int b = threadIdx.x; b < (E >> 4); b += 256) ext_quant(x + 16 * b, q + b, sx + b, corr + b);
}

/* lane partial of a row (k_gemv_q4b_dp4a_v2, CF:1688-1713: chunk c in lane c % 32), all of its bytes requested first */
template <int NIT> struct ExtRow { int4 w[NIT]; unsigned short sc[NIT]; };
template <int NIT>
__device__ __forceinline__ void ext_load(ExtRow<NIT> &r, const uint8_t *codes, const uint16_t *bs, int n32, int lane) {
#pragma unroll
    for (int i = 0; i < NIT; i++) {
        const int c = lane + 32 * i;
        if (c < n32) { r.w[i] = ld_stream16(codes + 16 * (size_t)c); r.sc[i] = ld_stream_u16(bs + c); }
    }
}
template <int NIT>
__device__ __forceinline__ float ext_dot(const ExtRow<NIT> &r, const int4 *q, const float *sx, const int *corr, int n32, int lane) {
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < NIT; i++) {
        const int c = lane + 32 * i;
        if (c < n32) {
            int a0, a1;
            q4b_chunk_dot(r.w[i], q[2 * c], q[2 * c + 1], corr[2 * c], corr[2 * c + 1], a0, a1);
            acc = __fmaf_rn(h2f(r.sc[i]), __fmaf_rn((float)a0, sx[2 * c], __fmul_rn((float)a1, sx[2 * c + 1])), acc);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    return acc;
}

struct ExtArgs {
    const uint8_t *g_codes, *u_codes, *d_codes; const uint16_t *g_bs, *u_bs, *d_bs;
    int E, FF; ExtPick pick;
    const int4 *qx; const float *sx; const int *cx;      /* x, quantised */
    float *h;                                            /* [picked][FF] silu(gate) * up */
    float *acc, *y; int first, last;                     /* [E] sums over earlier rounds; y: page-locked host memory */
};
/* one warp per (chosen expert, hidden unit): its gate and up rows, then (g / (1 + exp(-g))) * u (k_silu_mul, CF:1377-1383) */
template <int NIT>
__global__ void __launch_bounds__(kExtT) k_ext_up(const __grid_constant__ ExtArgs a) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int nb = a.E >> 4, n32 = a.E >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, total = a.pick.n * a.FF;
    int4 *q = reinterpret_cast<int4 *>(sm); float *sx = reinterpret_cast<float *>(q + nb); int *cx = reinterpret_cast<int *>(sx + nb);
    const size_t rb = (size_t)a.E / 2;
    ExtRow<NIT> g, u;
    auto load = [&](int p) {
        const int k = p / a.FF;
        const size_t row = (size_t)a.pick.idx[k] * a.FF + (p - k * a.FF);
        ext_load<NIT>(g, a.g_codes + row * rb, a.g_bs + row * n32, n32, lane);
        ext_load<NIT>(u, a.u_codes + row * rb, a.u_bs + row * n32, n32, lane);
    };
    int p = blockIdx.x * kExtW + warp;
    if (p < total) load(p);                              /* weights: requested before the quantised x exists */
    sp_pdl_wait();
    sp_pdl_next();
    for (int b = threadIdx.x; b < nb; b += kExtT) { q[b] = a.qx[b]; sx[b] = a.sx[b]; cx[b] = a.cx[b]; }
    __syncthreads();
    for (; p < total; p += gridDim.x * kExtW) {
        const float x = ext_dot<NIT>(g, q, sx, cx, n32, lane), up = ext_dot<NIT>(u, q, sx, cx, n32, lane);
        if (lane == 0) a.h[p] = __fmul_rn(__fdiv_rn(x, __fadd_rn(1.0f, expf(-x))), up);
        if (p + (int)gridDim.x * kExtW < total) load(p + gridDim.x * kExtW);
    }
}
/* one warp per output row: the down rows of all chosen experts, accumulated in the caller's order (dg_k_axpy: fused
 * multiply-add). Every CTA quantises the hidden vectors for itself. */
template <int NIT>
__global__ void __launch_bounds__(kExtT) k_ext_down(const __grid_constant__ ExtArgs a) {
    extern __shared__ __align__(16) unsigned char sm[];
    constexpr int R = NIT == 1 ? 8 : NIT == 2 ? 4 : 2;   /* expert rows in flight */
    const int fb = a.FF >> 4, nb = a.pick.n * fb, n32 = a.FF >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = a.pick.n;
    int4 *q = reinterpret_cast<int4 *>(sm); float *sx = reinterpret_cast<float *>(q + nb); int *cx = reinterpret_cast<int *>(sx + nb);
    const size_t rb = (size_t)a.FF / 2;
    ExtRow<NIT> r[R];
    auto load = [&](int j, int k0) {
#pragma unroll
        for (int k = 0; k < R; k++)
            if (k0 + k < n) {
                const size_t row = (size_t)a.pick.idx[k0 + k] * a.E + j;
                ext_load<NIT>(r[k], a.d_codes + row * rb, a.d_bs + row * n32, n32, lane);
            }
    };
    int j = blockIdx.x * kExtW + warp;
    if (j < a.E) load(j, 0);
    sp_pdl_wait();
    for (int b = threadIdx.x; b < nb; b += kExtT) ext_quant(a.h + 16 * b, q + b, sx + b, cx + b);
    __syncthreads();
    for (; j < a.E; j += gridDim.x * kExtW) {
        float acc = a.first ? 0.0f : a.acc[j];
        for (int k0 = 0; k0 < n; k0 += R) {
#pragma unroll
            for (int k = 0; k < R; k++)
                if (k0 + k < n) acc = __fmaf_rn(a.pick.wt[k0 + k], ext_dot<NIT>(r[k], q + (k0 + k) * fb, sx + (k0 + k) * fb, cx + (k0 + k) * fb, n32, lane), acc);
            if (k0 + R < n) load(j, k0 + R);
        }
        if (lane == 0) { if (a.last) a.y[j] = acc; else a.acc[j] = acc; }
        if (j + (int)gridDim.x * kExtW < a.E) load(j + gridDim.x * kExtW, 0);
    }
}

struct ExtLayer {
    std::string tag; int NE, FF, E;
    uint8_t *g_codes, *u_codes, *d_codes; uint16_t *g_bs, *u_bs, *d_bs;
};

int ext_fail(const char *msg) { sp_set_error(msg); return 1; }

}  // namespace

struct ExtScratch {
    float *hx, *hy;                                        /* page-locked x[E] and y[E] */
    float *h, *acc; int4 *qx; float *sx; int *cx;          /* hidden vectors [kExtSlots][FF], sums of earlier rounds [E], int8 x */
};
struct sp_moe_ext {
    int device;
    cudaStream_t st;
    std::vector<ExtLayer> layers;
    ExtScratch s;
    int cap_e, cap_ff, sms;
};

static void ext_free_scratch(ExtScratch &s) {
    if (s.hx) cudaFreeHost(s.hx);
    if (s.hy) cudaFreeHost(s.hy);
    void *ps[] = {s.h, s.acc, s.qx, s.sx, s.cx};
    for (void *p : ps) if (p) cudaFree(p);
    s = ExtScratch{};
}
/* all-or-nothing: on failure whatever was allocated is freed and `s` is left empty */
static bool ext_alloc_scratch(ExtScratch &s, int ce, int cf) {
    s = ExtScratch{};
    const bool ok =
        cudaMallocHost((void **)&s.hx, 4 * (size_t)ce) == cudaSuccess && cudaMallocHost((void **)&s.hy, 4 * (size_t)ce) == cudaSuccess &&
        cudaMalloc((void **)&s.h, 4 * (size_t)cf * kExtSlots) == cudaSuccess && cudaMalloc((void **)&s.acc, 4 * (size_t)ce) == cudaSuccess &&
        cudaMalloc((void **)&s.qx, (size_t)ce) == cudaSuccess && cudaMalloc((void **)&s.sx, 4 * (size_t)(ce / 16)) == cudaSuccess &&
        cudaMalloc((void **)&s.cx, 4 * (size_t)(ce / 16)) == cudaSuccess;
    if (!ok) { ext_free_scratch(s); cudaGetLastError(); }
    return ok;
}

typedef void (*ExtKernel)(ExtArgs);
static ExtKernel ext_up_for(int E) { const int n = (E / 32 + 31) / 32; return n <= 1 ? k_ext_up<1> : n == 2 ? k_ext_up<2> : n == 3 ? k_ext_up<3> : k_ext_up<4>; }
static ExtKernel ext_down_for(int FF) { const int n = (FF / 32 + 31) / 32; return n <= 1 ? k_ext_down<1> : n == 2 ? k_ext_down<2> : n == 3 ? k_ext_down<3> : k_ext_down<4>; }
static size_t ext_smem(int n) { return (size_t)n + 8 * (size_t)(n / 16); }        /* n quantised activations */
/* CTAs for `units` warps of work: two to an SM at most */
static int ext_grid(const sp_moe_ext *h, int units) { const int g = (units + kExtW - 1) / kExtW, most = 2 * h->sms; return g < most ? g : most; }
static cudaError_t ext_prepare() {                         /* per device: 16 experts of 4096 hidden units take 96 KB */
    cudaError_t e = cudaSuccess;
    for (int n = 1024; n <= 4096 && e == cudaSuccess; n += 1024) e = cudaFuncSetAttribute(ext_down_for(n), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ext_smem(kExtSlots * 4096));
    return e;
}

extern "C" int sp_moe_ext_open(int device, sp_moe_ext **out) {
    if (!out) return ext_fail("sp_moe_ext_open: NULL argument");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return ext_fail("sp_moe_ext_open: no CUDA device; this library has no CPU path"); }
    if (device < 0 || device >= ndev) return ext_fail("sp_moe_ext_open: device out of range");
    if (cudaSetDevice(device) != cudaSuccess) return ext_fail("sp_moe_ext_open: cudaSetDevice failed");
    sp_moe_ext *h = new sp_moe_ext();
    h->device = device; h->s = ExtScratch{}; h->cap_e = h->cap_ff = 0; h->sms = 1;
    cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device);
    if (ext_prepare() != cudaSuccess) { delete h; return ext_fail("sp_moe_ext_open: kernel attributes"); }
    if (cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) != cudaSuccess) { delete h; return ext_fail("sp_moe_ext_open: stream creation failed"); }
    *out = h;
    return 0;
}

extern "C" int sp_moe_ext_close(sp_moe_ext *h) {
    if (!h) return 0;
    cudaSetDevice(h->device);
    cudaStreamSynchronize(h->st);
    for (auto &l : h->layers) { void *ps[] = {l.g_codes, l.u_codes, l.d_codes, l.g_bs, l.u_bs, l.d_bs}; for (void *p : ps) cudaFree(p); }
    ext_free_scratch(h->s);
    cudaStreamDestroy(h->st);
    delete h;
    return 0;
}

extern "C" int sp_moe_ext_upload_experts(sp_moe_ext *h, const char *tag,
                                         const uint8_t *gate_codes, const uint16_t *gate_bs,
                                         const uint8_t *up_codes, const uint16_t *up_bs,
                                         const uint8_t *down_codes, const uint16_t *down_bs, int NE, int FF, int E) {
    if (!h || !tag || !gate_codes || !gate_bs || !up_codes || !up_bs || !down_codes || !down_bs) return ext_fail("sp_moe_ext_upload_experts: NULL argument");
    if (NE <= 0 || FF <= 0 || E <= 0 || (FF & 31) || (E & 31) || FF > 4096 || E > 4096) return ext_fail("sp_moe_ext_upload_experts: E and FF must be multiples of 32 in (0, 4096]");
    if (cudaSetDevice(h->device) != cudaSuccess) return ext_fail("sp_moe_ext_upload_experts: cudaSetDevice failed");
    ExtLayer l{}; l.tag = tag; l.NE = NE; l.FF = FF; l.E = E;
    const size_t gb = (size_t)NE * FF * E / 2, gs = (size_t)NE * FF * (E / 32) * 2, db = (size_t)NE * E * FF / 2, ds = (size_t)NE * E * (FF / 32) * 2;
    struct { void **p; const void *src; size_t n; } up[] = {{(void **)&l.g_codes, gate_codes, gb}, {(void **)&l.g_bs, gate_bs, gs}, {(void **)&l.u_codes, up_codes, gb},
                                                           {(void **)&l.u_bs, up_bs, gs}, {(void **)&l.d_codes, down_codes, db}, {(void **)&l.d_bs, down_bs, ds}};
    bool ok = true;
    for (auto &u : up) { *u.p = nullptr; if (ok && (cudaMalloc(u.p, u.n) != cudaSuccess || cudaMemcpy(*u.p, u.src, u.n, cudaMemcpyHostToDevice) != cudaSuccess)) ok = false; }
    if (ok && (E > h->cap_e || FF > h->cap_ff)) {          /* scratch for the largest shapes seen so far */
        /* the larger set is allocated first and swapped in only when it is complete: on failure the old
         * scratch, its sizes and the layers uploaded earlier all stay valid */
        const int ce = E > h->cap_e ? E : h->cap_e, cf = FF > h->cap_ff ? FF : h->cap_ff;
        ExtScratch fresh;
        ok = ext_alloc_scratch(fresh, ce, cf);
        if (ok) {
            cudaStreamSynchronize(h->st);
            ext_free_scratch(h->s);
            h->s = fresh; h->cap_e = ce; h->cap_ff = cf;
        }
    }
    if (!ok) {
        for (auto &u : up) if (*u.p) cudaFree(*u.p);
        cudaGetLastError();
        return ext_fail("sp_moe_ext_upload_experts: device allocation or copy failed");
    }
    h->layers.push_back(l);
    return 0;
}

extern "C" int sp_moe_ext_moe(void *vh, const char *tag, const int *idx, const float *wt, int NU,
                              const float *x, int E, int FF, float *y) {
    sp_moe_ext *h = (sp_moe_ext *)vh;
    if (!h || !tag || !idx || !wt || !x || !y || NU <= 0) return -1;
    const ExtLayer *M = nullptr;
    for (const auto &l : h->layers) if (l.tag == tag) { M = &l; break; }
    if (!M || M->FF != FF || M->E != E) return -1;                       /* not mine */
    for (int k = 0; k < NU; k++) if (idx[k] < 0 || idx[k] >= M->NE) { sp_set_error("sp_moe_ext_moe: expert index out of range"); return -1; }
    if (cudaSetDevice(h->device) != cudaSuccess) return -1;
    cudaStream_t st = h->st;
    memcpy(h->s.hx, x, 4 * (size_t)E);                                  /* the stream is idle between calls, also after one that failed */
    ExtArgs a{};
    a.g_codes = M->g_codes; a.u_codes = M->u_codes; a.d_codes = M->d_codes; a.g_bs = M->g_bs; a.u_bs = M->u_bs; a.d_bs = M->d_bs;
    a.E = E; a.FF = FF; a.qx = h->s.qx; a.sx = h->s.sx; a.cx = h->s.cx; a.h = h->s.h; a.acc = h->s.acc; a.y = h->s.hy;
    int nl = 0;
    cudaError_t e = sp_launch(k_ext_quant, dim3(1), 256, 0, st, &nl, h->s.hx, E, h->s.qx, h->s.sx, h->s.cx);
    for (int k0 = 0; k0 < NU && e == cudaSuccess; k0 += kExtSlots) {    /* one round unless a token has more than 16 experts */
        a.pick.n = NU - k0 < kExtSlots ? NU - k0 : kExtSlots;
        for (int k = 0; k < a.pick.n; k++) { a.pick.idx[k] = idx[k0 + k]; a.pick.wt[k] = wt[k0 + k]; }
        a.first = k0 == 0; a.last = k0 + kExtSlots >= NU;
        e = sp_launch(ext_up_for(E), dim3((unsigned)ext_grid(h, a.pick.n * FF)), kExtT, ext_smem(E), st, &nl, a);
        if (e == cudaSuccess) e = sp_launch(ext_down_for(FF), dim3((unsigned)ext_grid(h, E)), kExtT, ext_smem(a.pick.n * FF), st, &nl, a);
    }
    const cudaError_t done = cudaStreamSynchronize(st);                 /* what was launched still reads hx, also when a later launch failed */
    if (e != cudaSuccess || done != cudaSuccess) { cudaGetLastError(); sp_set_error("sp_moe_ext_moe: a kernel of the call failed"); return -1; }
    memcpy(y, h->s.hy, 4 * (size_t)E);
    return 0;
}
