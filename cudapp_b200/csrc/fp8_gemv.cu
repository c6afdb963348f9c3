// fp8_gemv.cu: FP8 e4m3 block-scaled GEMV / grouped GEMV / grouped row-table GEMM on the CUDA cores.
//
// This is the exactness engine: it keeps the summation order of the reference kernels
// (src/omega_blackwell_codegen_moe.h:13-29, src/omega_blackwell_codegen_gemm.h:5-14; host emulation
// tests/gpu_fp8gemm_test.c:48-69) so every output is bit-identical to them: lane L of a warp owns LB contiguous
// columns per K step of 32*LB columns; dot = FMA chain over those LB bytes; acc = fma(dot, scale, acc) once per
// step; lanes are summed by a shuffle-down tree 16, 8, 4, 2, 1. The reference folds 2^-120 / 2^64 / 2^56 into
// w / x / scale because its integer byte decode yields e4m3 * 2^-120; here cvt.f16x2.e4m3x2 decodes exactly, so
// no fold is stored (the folds are exact powers of two whose product is 1: same bits).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdlib.h>
#include "internal.h"

namespace b200 {

template <int LB> struct WVec;
template <> struct WVec<16> { using T = uint4; };
template <> struct WVec<8> { using T = uint2; };
template <> struct WVec<4> { using T = uint32_t; };

__device__ __forceinline__ void decode4(uint32_t v, float *o) {
    uint32_t lo, hi;
    asm("{ .reg .b16 a, b; mov.b32 {a, b}, %2; cvt.rn.f16x2.e4m3x2 %0, a; cvt.rn.f16x2.e4m3x2 %1, b; }" : "=r"(lo), "=r"(hi) : "r"(v));
    const float2 f0 = __half22float2(*reinterpret_cast<__half2 *>(&lo)), f1 = __half22float2(*reinterpret_cast<__half2 *>(&hi));
    o[0] = f0.x; o[1] = f0.y; o[2] = f1.x; o[3] = f1.y;
}
__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
// (q-th float4 of a lane's LB columns): the xor spreads the four float4 of neighbouring lanes over all banks when a row is written to shared memory
template <int LB> __device__ __forceinline__ uint32_t xs_at(uint32_t q, uint32_t lane) { return q * 32u + (lane ^ (q * (LB == 16 ? 2u : LB == 8 ? 4u : 0u))); }

// grid (ctas, groups or segments); 4 warps. A CTA puts MT activation rows of its segment into shared memory as f32, in the lanes' own column
// order, and its warps then stream weight rows against them: R consecutive output rows per warp, the weights of the next PF K steps in flight.
// Bound by HBM when a segment has a few rows (64 tokens x 8 picks, [1536, 2048]: 400 MB), by the FP32 pipe from about four rows per expert on.
// With one output row per warp and x read per row from global memory, as this kernel was, every product cost a load and a conversion beside its
// FMA; four rows share them here, and fma.rn.f32x2 runs two rows' chains (each its own IEEE chain: the same bits) in one instruction slot.
constexpr uint32_t ROWS_WARPS = 4;
template <int MT> constexpr uint32_t ROWS_CHUNK = MT == 8 ? 2048u : 4096u;   // columns of x resident at a time: at most 64 KB, so that three CTAs share an SM
constexpr uint32_t GEMV_CTAS = 8;   // of the one-row GEMV form on an SM: 64 registers a thread. Left to itself it took 74 to 80 and six fitted, so that grids up to eight ran in two waves
// One row per warp: a lane has 64 bytes of weights in flight at every lane width. Four K steps whatever the width, as this was, are only 16 bytes where k is not a multiple of 256.
// Both together, us with a cold L2, before -> now: 8 x [512, 3968] 38.9 -> 20.5, 5 x [768, 8192] 32.7 -> 23.3, 1 x [512, 8320] 42.9 -> 30.7, 3 x [1536, 4224] 43.0 -> 22.5. With four
// rows per warp two steps stay: 32 bytes per row at every width took up to 84 registers, one CTA per SM fewer (8 x [1536, 8320] 47 -> 75 us).
template <int LB, int R, int MT>
__global__ void __launch_bounds__(32 * ROWS_WARPS, MT == 1 ? (R == 1 ? GEMV_CTAS : 5) : 3) fp8_rows_kernel(const __grid_constant__ GemvArgs a) {
    griddep_chain();
    constexpr uint32_t STEP = 32u * LB, CS = ROWS_CHUNK<MT> / STEP, Q = LB / 4, NT = 32u * ROWS_WARPS;
    constexpr int PF = R == 1 ? 64 / LB : 2, PAIRS = R > 1 ? R / 2 : 1;
    using WT = typename WVec<LB>::T;
    extern __shared__ float4 xs[];                 // [step of the chunk][MT][Q][32]
    __shared__ const uint8_t *s_row[MT];
    const uint32_t g = blockIdx.y, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint64_t w_va, s_va; uint32_t row0, cnt;
    if (a.seg) {
        const Seg32 sg = a.seg[g];
        w_va = sg.w_va; s_va = sg.s_va; row0 = sg.row0; cnt = sg.cnt;
        if (cnt == 0) return;
    } else {
        const uint32_t gg = (a.mutant == 3 && (g ^ 1u) < a.groups_or_segs) ? (g ^ 1u) : g;
        w_va = a.tab ? a.tab[2 * gg] : a.tab_inline[2 * gg]; s_va = a.tab ? a.tab[2 * gg + 1] : a.tab_inline[2 * gg + 1]; row0 = g; cnt = 1;
    }
    const uint32_t n = a.n, k = a.k, kb = k / 128u, steps = k / STEP;
    const size_t xstride = a.x_stride_bytes ? a.x_stride_bytes : (size_t)k * (a.x_bf16 ? 2 : 4);
    for (uint32_t i0 = 0; i0 < cnt; i0 += MT) {
        const uint32_t mc = min((uint32_t)MT, cnt - i0);
        if (i0) __syncthreads();                   // the previous pass has read its rows
        if (tid < mc) {
            uint32_t p = row0 + i0 + tid;
            if (a.seg && a.mutant == 3 && (p ^ 1u) < a.rows) p ^= 1u;
            const uint32_t xi = a.seg ? (a.xmap ? a.xmap[p] : p) : (a.x_rows == 1 ? 0u : p);
            s_row[tid] = reinterpret_cast<const uint8_t *>(a.x) + (size_t)xi * xstride;
        }
        __syncthreads();
        auto stage = [&](uint32_t first) {         // columns [first, first + chunk) of the pass's rows
            const uint32_t cols = min(ROWS_CHUNK<MT>, k - first);
            for (uint32_t c = tid * 4u; c < cols; c += NT * 4u) {
                float4 v[MT];
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    v[m] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if ((uint32_t)m >= mc) continue;
                    if (a.x_bf16) {
                        const uint2 u = *reinterpret_cast<const uint2 *>(s_row[m] + (size_t)(first + c) * 2);
                        v[m] = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
                    } else v[m] = *reinterpret_cast<const float4 *>(s_row[m] + (size_t)(first + c) * 4);
                }
                const uint32_t st = c / STEP, rem = c % STEP;
                float4 *to = xs + (size_t)st * MT * Q * 32u + xs_at<LB>((rem % LB) / 4u, rem / LB);
#pragma unroll
                for (int m = 0; m < MT; m++) if ((uint32_t)m < ((mc + 1u) & ~1u) || MT == 1) to[m * Q * 32] = v[m];
            }
            __syncthreads();
        };
        const bool resident = k <= ROWS_CHUNK<MT>;
        WT raw[PF][R]; float sc[PF];
        auto fetch = [&](int slot, uint32_t rb, uint32_t st) {
            const uint8_t *wrow = reinterpret_cast<const uint8_t *>(w_va) + (size_t)rb * k + lane * LB;
            const float *srow = reinterpret_cast<const float *>(s_va) + (size_t)(rb / 128u) * kb;   // R divides 128: the R rows share a scale row
#pragma unroll
            for (int j = 0; j < R; j++) raw[slot][j] = __ldcs(reinterpret_cast<const WT *>(wrow + (size_t)j * k + (size_t)st * STEP));   // streaming: read once
            sc[slot] = a.mutant == 1 ? 1.0f : __ldg(srow + (a.mutant == 2 ? 0u : (st * STEP + lane * LB) / 128u));
        };
        const uint32_t rb0 = (blockIdx.x * ROWS_WARPS + warp) * R;
#pragma unroll
        for (int i = 0; i < PF; i++) if ((uint32_t)i < steps && rb0 < n) fetch(i, rb0, i);   // on its way while x is staged
        if (resident) stage(0);
        for (uint32_t rb = rb0; rb < n; rb += gridDim.x * ROWS_WARPS * R) {   // n is a multiple of 4 R: every warp makes the same number of turns
            uint64_t acc[MT][PAIRS];               // R > 1: two rows each; R = 1: the low half
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int p = 0; p < PAIRS; p++) acc[m][p] = 0;
            for (uint32_t st0 = 0; st0 < steps; st0 += PF) {
#pragma unroll
                for (int i = 0; i < PF; i++) {
                    const uint32_t st = st0 + i;
                    if (st >= steps) break;
                    if (!resident && st % CS == 0) { if (st || rb >= gridDim.x * ROWS_WARPS * R) __syncthreads(); stage(st * STEP); }
                    float wv[R][LB];
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        const uint32_t *u = reinterpret_cast<const uint32_t *>(&raw[i][j]);
#pragma unroll
                        for (int b = 0; b < LB / 4; b++) decode4(u[b], wv[j] + 4 * b);
                    }
                    const float s = sc[i];
                    // this slot's next weights: of this row group, or the first ones of the group after it
                    const bool more = st + PF < steps;
                    const uint32_t nrb = more ? rb : rb + gridDim.x * ROWS_WARPS * R;
                    if (nrb < n) fetch(i, nrb, more ? st + PF : (uint32_t)i);
                    const float4 *xst = xs + (size_t)(st % CS) * MT * Q * 32u;
#pragma unroll
                    for (int m0 = 0; m0 < MT; m0 += 2) {
                        if ((uint32_t)m0 >= mc) break;
#pragma unroll
                        for (int m = m0; m < (m0 + 2 < MT ? m0 + 2 : MT); m++) {
                            float xv[LB];
#pragma unroll
                            for (int q = 0; q < (int)Q; q++) *reinterpret_cast<float4 *>(xv + 4 * q) = xst[m * Q * 32 + xs_at<LB>(q, lane)];
                            if constexpr (R > 1) {
#pragma unroll
                                for (int p = 0; p < PAIRS; p++) {
                                    uint64_t dot = 0;
#pragma unroll
                                    for (int b = 0; b < LB; b++) dot = fma2(pack2(wv[2 * p][b], wv[2 * p + 1][b]), pack2(xv[b], xv[b]), dot);
                                    acc[m][p] = fma2(dot, pack2(s, s), acc[m][p]);
                                }
                            } else {
                                float dot = 0.0f;
#pragma unroll
                                for (int b = 0; b < LB; b++) dot = fmaf(wv[0][b], xv[b], dot);
                                acc[m][0] = pack2(fmaf(dot, s, __uint_as_float((uint32_t)acc[m][0])), 0.0f);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < MT; m++) {
                if ((uint32_t)m >= mc) break;
                float v[R];
#pragma unroll
                for (int p = 0; p < PAIRS; p++) { v[R > 1 ? 2 * p : 0] = __uint_as_float((uint32_t)acc[m][p]); if (R > 1) v[R > 1 ? 2 * p + 1 : 0] = __uint_as_float((uint32_t)(acc[m][p] >> 32)); }
                // the shuffle-down tree's lane-0 sum: an exchange adds the same pairs (addition commutes), and with four rows the first two exchanges also
                // deal the rows to the lane quarters, so the tree costs 6 shuffles instead of 20 and the four results leave as one 16-byte run
                float t; uint32_t j = 0; bool out = lane == 0;
                if constexpr (R == 4) {
                    const bool h16 = lane & 16u, h8 = lane & 8u;
                    const float a0 = (h16 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[2], 16), a1 = (h16 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[3], 16);
                    t = (h8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, h8 ? a0 : a1, 8);
                    j = (h16 ? 2u : 0u) + (h8 ? 1u : 0u); out = (lane & 7u) == 0;
                } else {
                    t = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
                    t += __shfl_xor_sync(0xffffffffu, t, 8);
                }
                t += __shfl_xor_sync(0xffffffffu, t, 4); t += __shfl_xor_sync(0xffffffffu, t, 2); t += __shfl_xor_sync(0xffffffffu, t, 1);
                if (out) {
                    const uint32_t p = row0 + i0 + m, yi = (a.seg && a.ymap) ? a.ymap[p] : p;
                    a.y[(size_t)yi * n + rb + j] = t * a.out_mul;
                }
            }
        }
    }
}

template <int LB, int R, int MT>
static cudaError_t launch_one(const GemvArgs &a, dim3 grid, cudaStream_t s) {
    const size_t smem = (size_t)MT * (a.k < ROWS_CHUNK<MT> ? a.k : ROWS_CHUNK<MT>) * 4;
    if (smem > 40 * 1024) {   // near 48 KB with the static words; set on every call: it belongs to the device's context, and a failure must not outlive its call
        const cudaError_t e = cudaFuncSetAttribute(fp8_rows_kernel<LB, R, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(MT * ROWS_CHUNK<MT> * 4));
        if (e != cudaSuccess) return e;
    }
    return launch_chained(fp8_rows_kernel<LB, R, MT>, grid, dim3(32 * ROWS_WARPS), smem, s, a);
}
template <int R, int MT>
static cudaError_t launch_lb(const GemvArgs &a, dim3 grid, cudaStream_t s) {
    const uint32_t k = a.k;
    if (k % 512u == 0) return launch_one<16, R, MT>(a, grid, s);
    if (k % 256u == 0) return launch_one<8, R, MT>(a, grid, s);
    return launch_one<4, R, MT>(a, grid, s);
}

// GEMV forms: one activation row per group. One row per warp while all of its CTAs are resident at once, else four rows per warp (a quarter of the CTAs,
// each x value read once for four products). A row's arithmetic does not depend on how rows are dealt to warps: same bits.
cudaError_t launch_gemv_grouped(const GemvArgs &a, uint32_t cta_budget, uint32_t *grid_x, uint32_t *warps, cudaStream_t s) {
    const uint32_t sms = st().sm_count ? st().sm_count : 148u;
    const bool few = (uint64_t)(a.n / ROWS_WARPS) * a.groups_or_segs <= GEMV_CTAS * sms && !cta_budget;
    uint32_t gx = few ? a.n / ROWS_WARPS : a.n / (4u * ROWS_WARPS);
    if (cta_budget && gx > cta_budget) gx = cta_budget;
    if (warps) *warps = ROWS_WARPS;
    if (grid_x) *grid_x = gx;
    return few ? launch_lb<1, 1>(a, dim3(gx, a.groups_or_segs), s) : launch_lb<4, 1>(a, dim3(gx, a.groups_or_segs), s);
}
static uint32_t gemm_rows_mt(uint32_t k) { return k <= ROWS_CHUNK<8> ? 8u : 4u; }
// Row-table form: up to eight activation rows per pass of a segment's weights (four where eight rows of x would leave room for one CTA per SM).
// A CTA keeps its rows of x for several 16-row weight groups: about twelve CTAs per SM in all (three at a time), so that long and short segments even out.
cudaError_t launch_gemm_rows(const GemvArgs &a, uint32_t *grid_x, uint32_t *mt, cudaStream_t s) {
    const uint32_t sms = st().sm_count ? st().sm_count : 148u, groups = a.n / (4u * ROWS_WARPS), want = (sms * 12u + a.groups_or_segs - 1u) / a.groups_or_segs;
    const uint32_t per = (groups + want - 1u) / want, gx = (groups + per - 1u) / per, rows = gemm_rows_mt(a.k);
    if (grid_x) *grid_x = gx;
    if (mt) *mt = rows;
    return rows == 8u ? launch_lb<4, 8>(a, dim3(gx, a.groups_or_segs), s) : launch_lb<4, 4>(a, dim3(gx, a.groups_or_segs), s);
}

// ---------------------------------------------------------------- host-staged API cores
static void fill_info(OmegaGpuFp8Info *info, const OmegaGpuFp8Tensor *t, uint32_t groups, uint32_t gx, uint32_t warps) {
    if (!info) return;
    const uint32_t lb = t->k % 512u == 0 ? 16u : t->k % 256u == 0 ? 8u : 4u;
    info->experts = t->experts; info->n = t->n; info->k = t->k; info->groups = groups;
    info->lane_bytes = lb; info->rows_per_warp = 4; info->warps_per_cta = warps; info->depth = 0;
    info->grid_x = gx; info->grid_y = groups; info->steps = t->k / (32u * lb);
    info->weight_bytes = (uint64_t)groups * t->n * t->k;
    info->scale_bytes = (uint64_t)groups * (t->n / 128u) * (t->k / 128u) * 4u;
    info->kernel_cache_hit = true;
    snprintf(info->target_chip, sizeof info->target_chip, "%s", st().chip);
    info->sm_architecture = 100;
    info->general = lb == 4u || groups > OMEGA_GPU_FP8_MAX_GROUPS;
}

// whether a result still holds the poison it was filled with: sets a flag in mapped host memory
__global__ void __launch_bounds__(256) poison_scan_kernel(const float4 *__restrict__ y, size_t n4, uint32_t *flag) {
    bool bad = false;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += (size_t)gridDim.x * 256) {
        const float4 v = __ldg(y + i);
        bad |= v.x == POISON_F32 || v.y == POISON_F32 || v.z == POISON_F32 || v.w == POISON_F32;
    }
    if (bad) *flag = 1;
}

// A host call's result. Up to RESULT_BYTES the kernel stores it straight into mapped host memory, which was filled with poison before the launch: the
// host takes each word as soon as it is no longer poison, and the call pays neither a fill kernel nor a copy nor a stream synchronisation (a single
// [768, 2048] projection called from Python, binding included: 49 -> 19 us). Larger results are poisoned, scanned and copied from device memory.
struct HostResult {
    float *dev = nullptr; volatile float *mapped = nullptr; void *area = nullptr; size_t count; cudaStream_t s;
    bool open(size_t words, cudaStream_t stream) {
        count = words; s = stream; area = result_area();
        if (!area) return false;
        if (words * 4 <= RESULT_BYTES) {
            mapped = (volatile float *)area;
            for (size_t i = 0; i < words; i++) mapped[i] = POISON_F32;
            dev = (float *)area;   // unified addressing: the host's pointer is the device's
            return true;
        }
        dev = (float *)stage(2, words * 4);
        if (dev) launch_fill_f32(dev, words, POISON_F32, s);
        return dev != nullptr;
    }
    // 0, or CHIP_FAIL with the error text set; y is written only when every word was produced. sync: the caller reads events afterwards
    int take(float *y, bool sync, const char *what) {
        bool left = false;
        if (mapped) {
            if (!sync) {   // bounded: past the limit the stream decides (a fault, a result word that equals the poison)
                const uint64_t until = now_ns() + 2000000;
                for (size_t i = 0; i < count; i++)
                    for (uint32_t spin = 1; mapped[i] == POISON_F32; spin++)
                        if (spin % 1024 == 0 && now_ns() > until) { sync = true; i = count - 1; break; }
            }
            if (sync && !cuda_ok(cudaStreamSynchronize(s), what)) return OMEGA_GPU_FP8_CHIP_FAIL;
            if (sync) for (size_t i = 0; i < count; i++) left |= mapped[i] == POISON_F32;
            if (!left) memcpy(y, area, count * 4);
        } else {
            volatile uint32_t *flag = result_flag(area);
            *flag = 0;
            const size_t blocks = (count / 4 + 255) / 256;
            poison_scan_kernel<<<(unsigned)(blocks < 592 ? blocks : 592), 256, 0, s>>>((const float4 *)dev, count / 4, (uint32_t *)flag);   // count: rows of a multiple of 128 values
            if (!cuda_ok(cudaGetLastError(), "poison scan launch") || !to_host(y, dev, count * 4, s, flag) || !cuda_ok(cudaStreamSynchronize(s), what)) return OMEGA_GPU_FP8_CHIP_FAIL;
            left = *flag != 0;
        }
        if (left) { set_error("output poison survived"); return OMEGA_GPU_FP8_CHIP_FAIL; }
        return OMEGA_GPU_FP8_OK;
    }
};

// host bytes of one call; no exception may leave a C entry, so it is malloc's memory
struct HostBytes {
    char *p; size_t bytes;
    explicit HostBytes(size_t n) : p((char *)malloc(n)), bytes(n) {}
    ~HostBytes() { free(p); }
    HostBytes(const HostBytes &) = delete;
};

// ids / x on the host, or tab / x on the device (dev form). y always a host buffer here.
static int gemv_core(const OmegaGpuFp8Tensor *t, uint32_t groups, const uint32_t *ids, const float *x32, const uint16_t *x16,
                     uint32_t x_rows, float *y, OmegaGpuFp8Info *info, uint64_t dev_tab, uint64_t dev_x) {
    const uint64_t t0 = now_ns();
    if (info) memset(info, 0, sizeof *info);
    if (!t || !t->w || (!ids && !dev_tab) || (!x32 && !x16 && !dev_x) || !y || groups == 0 || (x_rows != 1 && x_rows != groups)) return OMEGA_GPU_FP8_BAD_ARGS;
    if (!dev_tab) for (uint32_t g = 0; g < groups; g++) if (ids[g] >= t->experts) return OMEGA_GPU_FP8_BAD_ARGS;
    if (dev_tab && groups > OMEGA_GPU_FP8_MAX_GROUPS) return OMEGA_GPU_FP8_TOO_LARGE;
    Lock l;
    State &g = st();
    if (!dev_open()) return OMEGA_GPU_FP8_CHIP_FAIL;
    const uint32_t n = t->n, k = t->k;
    cudaStream_t s = g.stream;
    GemvArgs a = {};
    if (dev_tab) a.tab = (const uint64_t *)(uintptr_t)dev_tab;
    else if (groups <= sizeof a.tab_inline / 16) for (uint32_t i = 0; i < groups; i++) (void)omega_gpu_fp8_tensor_entry(t, ids[i], &a.tab_inline[2 * i], &a.tab_inline[2 * i + 1]);
    else {
        HostBytes table((size_t)groups * 16);
        uint64_t *ht = (uint64_t *)table.p, *tab = (uint64_t *)stage(0, table.bytes);
        if (!ht) return OMEGA_GPU_FP8_BAD_ARGS;
        for (uint32_t i = 0; i < groups; i++) (void)omega_gpu_fp8_tensor_entry(t, ids[i], &ht[2 * i], &ht[2 * i + 1]);
        if (!tab || !to_device(tab, ht, table.bytes, s)) return OMEGA_GPU_FP8_CHIP_FAIL;
        a.tab = tab;
    }
    if (!dev_x) {
        const size_t xbytes = (size_t)x_rows * k * (x16 ? 2 : 4);
        void *xd = stage(1, xbytes);
        if (!xd || !to_device(xd, x32 ? (const void *)x32 : (const void *)x16, xbytes, s)) return OMEGA_GPU_FP8_CHIP_FAIL;
        a.x = xd;
    } else a.x = (const void *)(uintptr_t)dev_x;
    HostResult r;
    if (!r.open((size_t)groups * n, s)) return OMEGA_GPU_FP8_CHIP_FAIL;
    a.x_bf16 = (!dev_x && x16) ? 1 : 0; a.x_rows = x_rows;
    a.y = r.dev; a.n = n; a.k = k; a.groups_or_segs = groups; a.rows = groups;
    a.out_mul = dev_x ? 5.421010862427522e-20f /* 2^-64: the reference router's fold on x' */ : 1.0f;
    a.mutant = g.gemv_mutant;
    uint32_t gx = 0, warps = 0;
    if (info) cudaEventRecord(g.ev0, s);
    bool ok = cuda_ok(launch_gemv_grouped(a, g.cta_budget, &gx, &warps, s), "gemv launch");
    if (info) cudaEventRecord(g.ev1, s);
    const int rc = ok ? r.take(y, info != nullptr, "gemv") : OMEGA_GPU_FP8_CHIP_FAIL;
    fill_info(info, t, groups, gx, warps);
    if (info && ok) { float ms = 0; if (cudaEventElapsedTime(&ms, g.ev0, g.ev1) == cudaSuccess) info->elapsed_ns = (uint64_t)(ms * 1e6); info->completion_marker = 1; }
    if (info) info->call_ns = now_ns() - t0;
    return rc;
}

static int gemm_core(const OmegaGpuFp8Tensor *t, uint32_t M, const uint32_t *ids, const uint32_t *trow, const float *x32, const uint16_t *x16,
                     uint32_t x_rows, float *y, OmegaGpuFp8GemmInfo *info) {
    const uint64_t t0 = now_ns();
    if (info) memset(info, 0, sizeof *info);
    if (!t || !t->experts || !ids || !trow || (!x32 && !x16) || !y || M == 0 || x_rows == 0) return OMEGA_GPU_FP8GEMM_BAD_ARGS;
    uint32_t segs = 0;
    for (uint32_t i = 0; i < M; i++) {
        if (ids[i] >= t->experts || trow[i] >= x_rows || (i && ids[i] < ids[i - 1])) return OMEGA_GPU_FP8GEMM_BAD_ARGS;
        if (i == 0 || ids[i] != ids[i - 1]) segs++;
    }
    Lock l;
    State &g = st();
    if (!dev_open()) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    const uint32_t n = t->n, k = t->k;
    const size_t xbytes = (size_t)x_rows * k * (x16 ? 2 : 4), sbytes = (size_t)segs * sizeof(Seg32);
    HostBytes tables(sbytes + (size_t)M * 4);   // segment records, then the row table: one copy
    if (!tables.p) return OMEGA_GPU_FP8GEMM_BAD_ARGS;
    Seg32 *hseg = (Seg32 *)tables.p;
    memcpy(tables.p + sbytes, trow, (size_t)M * 4);
    uint32_t sg = 0; uint64_t passes = 0, passes_max = 0;
    const uint32_t mt = gemm_rows_mt(k);
    for (uint32_t i = 0; i < M;) {
        uint32_t j = i; while (j < M && ids[j] == ids[i]) j++;
        (void)omega_gpu_fp8_tensor_entry(t, ids[i], &hseg[sg].w_va, &hseg[sg].s_va);
        hseg[sg].row0 = i; hseg[sg].cnt = j - i; hseg[sg].pad = 0;
        const uint32_t p = (j - i + mt - 1u) / mt; if (p > passes_max) passes_max = p;
        passes += p;
        sg++; i = j;
    }
    cudaStream_t s = g.stream;
    char *dt = (char *)stage(0, tables.bytes); void *xd = stage(1, xbytes);
    HostResult r;
    if (!dt || !xd || !to_device(dt, tables.p, tables.bytes, s) || !to_device(xd, x32 ? (const void *)x32 : (const void *)x16, xbytes, s) ||
        !r.open((size_t)M * n, s)) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    GemvArgs a = {};
    a.seg = (const Seg32 *)dt; a.x = xd; a.x_bf16 = x16 ? 1 : 0; a.x_rows = x_rows; a.xmap = (const uint32_t *)(dt + sbytes); a.ymap = nullptr;
    a.y = r.dev; a.n = n; a.k = k; a.groups_or_segs = segs; a.rows = M; a.out_mul = 1.0f; a.mutant = g.gemm_mutant;
    uint32_t gx = 0;
    if (info) cudaEventRecord(g.ev0, s);
    const bool ok = cuda_ok(launch_gemm_rows(a, &gx, nullptr, s), "fp8gemm launch");
    if (info) cudaEventRecord(g.ev1, s);
    const int rc = ok ? r.take(y, info != nullptr, "fp8gemm") : OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    if (info) {
        const uint32_t lb = k % 512u == 0 ? 16u : k % 256u == 0 ? 8u : 4u;
        info->rows = M; info->segments = segs; info->n = n; info->k = k; info->mt = mt; info->warps_per_cta = ROWS_WARPS; info->lane_bytes = lb;
        info->grid_x = gx; info->grid_y = segs; info->passes_max = (uint32_t)passes_max;
        info->weight_bytes = (uint64_t)segs * n * k; info->streamed_bytes = passes * n * k; info->kernel_cache_hit = true;
        info->general = lb == 4u;
        if (ok) { float ms = 0; if (cudaEventElapsedTime(&ms, g.ev0, g.ev1) == cudaSuccess) info->elapsed_ns = (uint64_t)(ms * 1e6); info->completion_marker = 1; }
        info->call_ns = now_ns() - t0;
    }
    return rc;
}


// ---------------------------------------------------------------- allocation-free row-table GEMM
// The segment table the grouped GEMM kernel reads normally lives in a cudaMalloc'ed staging buffer. This variant
// keeps it in a fixed device array instead, so the whole call touches no allocator. Layout of the array:
// [0, 32 * NOALLOC_MAX_SEGMENTS) segment records, then one 16-byte header {segments, status, 0, 0}.
constexpr uint32_t NOALLOC_MAX_SEGMENTS = OMEGA_GPU_FP8GEMM_NOALLOC_MAX_SEGMENTS;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_MAX_SEGMENTS * 32 + 256];
static void *g_noalloc_ptr[64];   // per device: the array's DEVICE address (the symbol itself is only a host-side stand-in)

// One CTA. Turns M sorted expert ids into segment records {w_va, s_va, row0, cnt}. status: 0 ok, 1 ids not sorted or
// out of range, 2 more segments than the table holds, 3 an activation row index at or past x_rows (the GEMM kernel would
// read x out of bounds). Everything a previous call left behind is overwritten: the header is rewritten, records
// [segments, max) are zeroed.
__global__ void __launch_bounds__(1024) noalloc_segments_kernel(unsigned char *scratch, uint32_t M, uint32_t experts, const uint32_t *__restrict__ ids,
                                                                const uint32_t *__restrict__ token_rows, uint32_t x_rows,
                                                                uint64_t w_base, uint64_t s_base, uint64_t w_stride, uint64_t s_stride) {
    __shared__ uint32_t warp_sum[32];
    __shared__ uint32_t s_run, s_bad, s_bad_row;
    Seg32 *seg = reinterpret_cast<Seg32 *>(scratch);
    uint32_t *hdr = reinterpret_cast<uint32_t *>(scratch + NOALLOC_MAX_SEGMENTS * 32);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) { s_run = 0; s_bad = 0; s_bad_row = 0; }
    __syncthreads();
    for (uint32_t base = 0; base < M; base += 1024) {
        const uint32_t i = base + tid;
        uint32_t flag = 0, e = 0;
        if (i < M) {
            e = ids[i];
            if (token_rows[i] >= x_rows) s_bad_row = 1;
            const uint32_t prev = i ? ids[i - 1] : 0xffffffffu;
            if (e >= experts || (i && e < prev)) s_bad = 1;
            flag = (i == 0 || e != prev) ? 1u : 0u;
        }
        uint32_t inc = flag;
        for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= (uint32_t)o) inc += u; }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        uint32_t before = s_run;
        for (uint32_t w = 0; w < warp; w++) before += warp_sum[w];
        const uint32_t si = before + inc - flag;
        if (flag && si < NOALLOC_MAX_SEGMENTS && e < experts) {
            Seg32 r; r.w_va = w_base + (uint64_t)e * w_stride; r.s_va = s_base + (uint64_t)e * s_stride; r.row0 = i; r.cnt = 0; r.pad = 0;
            seg[si] = r;
        }
        __syncthreads();
        if (tid == 0) { uint32_t tot = 0; for (int w = 0; w < 32; w++) tot += warp_sum[w]; s_run += tot; }
        __syncthreads();
    }
    const uint32_t S = s_run, kept = min(S, NOALLOC_MAX_SEGMENTS);
    for (uint32_t z = tid; z < kept; z += 1024) seg[z].cnt = (z + 1 < kept ? seg[z + 1].row0 : M) - seg[z].row0;
    for (uint32_t z = kept + tid; z < NOALLOC_MAX_SEGMENTS; z += 1024) { const Seg32 zero = {0, 0, 0, 0, 0}; seg[z] = zero; }
    if (tid == 0) { hdr[0] = kept; hdr[1] = s_bad ? 1u : (s_bad_row ? 3u : (S > NOALLOC_MAX_SEGMENTS ? 2u : 0u)); hdr[2] = 0; hdr[3] = 0; }
}

}  // namespace b200
using namespace b200;

extern "C" {
int omega_gpu_fp8_gemv_f32(const OmegaGpuFp8Tensor *t, uint32_t expert, const float *x, float *y, OmegaGpuFp8Info *info) {
    return gemv_core(t, 1, &expert, x, nullptr, 1, y, info, 0, 0);
}
int omega_gpu_fp8_gemv_bf16(const OmegaGpuFp8Tensor *t, uint32_t expert, const uint16_t *x, float *y, OmegaGpuFp8Info *info) {
    return gemv_core(t, 1, &expert, nullptr, x, 1, y, info, 0, 0);
}
int omega_gpu_fp8_gemv_grouped_f32(const OmegaGpuFp8Tensor *t, uint32_t groups, const uint32_t *ids, const float *x, uint32_t x_rows, float *y, OmegaGpuFp8Info *info) {
    return gemv_core(t, groups, ids, x, nullptr, x_rows, y, info, 0, 0);
}
int omega_gpu_fp8_gemv_grouped_dev(const OmegaGpuFp8Tensor *t, uint32_t groups, uint64_t tab_va, uint64_t x_va, float *y, OmegaGpuFp8Info *info) {
    if (!tab_va || !x_va) return OMEGA_GPU_FP8_BAD_ARGS;
    return gemv_core(t, groups, nullptr, nullptr, nullptr, 1, y, info, tab_va, x_va);
}
int omega_gpu_fp8_gemv_grouped_async(const OmegaGpuFp8Tensor *t, uint32_t groups, uint64_t tab_va, uint64_t x_va, uint32_t x_rows, int x_bf16,
                                     uint64_t y_va, void *stream) {
    if (!t || !tab_va || !x_va || !y_va || groups == 0 || (x_rows != 1 && x_rows != groups)) return OMEGA_GPU_FP8_BAD_ARGS;
    if (!st().opened || st().latched) return OMEGA_GPU_FP8_CHIP_FAIL;
    GemvArgs a = {};
    a.tab = (const uint64_t *)(uintptr_t)tab_va; a.x = (const void *)(uintptr_t)x_va; a.x_bf16 = x_bf16; a.x_rows = x_rows;
    a.y = (float *)(uintptr_t)y_va; a.n = t->n; a.k = t->k; a.groups_or_segs = groups; a.rows = groups; a.out_mul = 1.0f;
    return cuda_ok(launch_gemv_grouped(a, 0, nullptr, nullptr, (cudaStream_t)stream), "gemv launch") ? OMEGA_GPU_FP8_OK : OMEGA_GPU_FP8_CHIP_FAIL;
}
int omega_gpu_fp8gemm_f32(const OmegaGpuFp8Tensor *t, uint32_t M, const uint32_t *ids, const uint32_t *trow, const float *x, uint32_t x_rows, float *y, OmegaGpuFp8GemmInfo *info) {
    return gemm_core(t, M, ids, trow, x, nullptr, x_rows, y, info);
}
int omega_gpu_fp8gemm_bf16(const OmegaGpuFp8Tensor *t, uint32_t M, const uint32_t *ids, const uint32_t *trow, const uint16_t *x, uint32_t x_rows, float *y, OmegaGpuFp8GemmInfo *info) {
    return gemm_core(t, M, ids, trow, nullptr, x, x_rows, y, info);
}
int omega_gpu_fp8gemm_async(const OmegaGpuFp8Tensor *t, uint32_t rows, uint32_t segs, uint64_t seg_va, uint64_t x_va, int x_bf16, uint64_t y_va,
                            uint64_t xmap_va, uint64_t ymap_va, void *stream) {
    if (!t || !seg_va || !x_va || !y_va || rows == 0 || segs == 0 || (!xmap_va != !ymap_va)) return OMEGA_GPU_FP8GEMM_BAD_ARGS;
    if (!st().opened || st().latched) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    GemvArgs a = {};
    a.seg = (const Seg32 *)(uintptr_t)seg_va; a.x = (const void *)(uintptr_t)x_va; a.x_bf16 = x_bf16; a.x_rows = rows;
    a.xmap = (const uint32_t *)(uintptr_t)xmap_va; a.ymap = (const uint32_t *)(uintptr_t)ymap_va;
    a.y = (float *)(uintptr_t)y_va; a.n = t->n; a.k = t->k; a.groups_or_segs = segs; a.rows = rows; a.out_mul = 1.0f;
    return cuda_ok(launch_gemm_rows(a, nullptr, nullptr, (cudaStream_t)stream), "fp8gemm launch") ? OMEGA_GPU_FP8GEMM_OK : OMEGA_GPU_FP8GEMM_CHIP_FAIL;
}

// Allocation-free entry (declared in b200moe_fp8gemm.h). Some hosts of this library may not allocate device memory
// at all once they are running: a serving process that has handed every byte to its own arena, a caller inside a
// latency-critical section, a plugin whose embedder forbids cudaMalloc after start-up. The host-staged calls above
// grow staging buffers on demand, so they are closed to such callers; this one is not. Every call blocks once on
// `stream` (it reads the table builder's status word back), so no call may be made while `stream` is being captured:
// such a call is refused with BAD_ARGS and queues nothing.
int omega_gpu_fp8gemm_noalloc(const OmegaGpuFp8Tensor *t, uint32_t M, uint64_t expert_ids_va, uint64_t token_rows_va, uint64_t x_va, int x_bf16,
                              uint32_t x_rows, uint64_t y_va, void *stream) {
    if (!t || !t->w || !M || !expert_ids_va || !token_rows_va || !x_va || !y_va || !x_rows) return OMEGA_GPU_FP8GEMM_BAD_ARGS;
    if (t->experts > NOALLOC_MAX_SEGMENTS) {
        set_error("fp8gemm_noalloc: the tensor has %u experts but the fixed segment table holds %u segments", t->experts, NOALLOC_MAX_SEGMENTS);
        return OMEGA_GPU_FP8GEMM_TOO_LARGE;
    }
    if (M > OMEGA_GPU_FP8GEMM_NOALLOC_MAX_ROWS) {
        set_error("fp8gemm_noalloc: %u rows is past the stated maximum of %u", M, OMEGA_GPU_FP8GEMM_NOALLOC_MAX_ROWS);
        return OMEGA_GPU_FP8GEMM_TOO_LARGE;
    }
    Lock l;
    State &g = st();
    if (!g.opened || g.latched) { set_error("fp8gemm_noalloc: the device is not open (upload a tensor first)"); return OMEGA_GPU_FP8GEMM_CHIP_FAIL; }
    if (t->device < 0 || t->device >= 64) return OMEGA_GPU_FP8GEMM_BAD_ARGS;
    cudaStream_t s = (cudaStream_t)stream;
    // every call waits once on `stream` for its table-building kernel, which a capturing stream cannot do: refuse before
    // anything is queued, so the caller's capture stays valid and nothing latches
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) { (void)cudaGetLastError(); set_error("fp8gemm_noalloc: not a usable stream"); return OMEGA_GPU_FP8GEMM_BAD_ARGS; }
    if (cap != cudaStreamCaptureStatusNone) { set_error("fp8gemm_noalloc: the stream is being captured; this entry synchronises the stream once per call and cannot be captured"); return OMEGA_GPU_FP8GEMM_BAD_ARGS; }
    if (!cuda_ok(cudaSetDevice(t->device), "cudaSetDevice")) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    if (!g_noalloc_ptr[t->device]) {   // set-up, once per device, with that device current
        void *p = nullptr;
        if (!cuda_ok(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress(noalloc scratch)") || !p) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
        g_noalloc_ptr[t->device] = p;
    }
    unsigned char *scratch = (unsigned char *)g_noalloc_ptr[t->device];
    uint64_t w0 = 0, s0 = 0;
    (void)omega_gpu_fp8_tensor_entry(t, 0, &w0, &s0);
    noalloc_segments_kernel<<<1, 1024, 0, s>>>(scratch, M, t->experts, (const uint32_t *)(uintptr_t)expert_ids_va,
                                               (const uint32_t *)(uintptr_t)token_rows_va, x_rows, w0, s0, (uint64_t)t->n * t->k,
                                               (uint64_t)(t->n / 128u) * (t->k / 128u) * 4u);
    if (!cuda_ok(cudaGetLastError(), "noalloc segments launch")) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    uint32_t hdr[4] = {0, 0, 0, 0};
    if (!cuda_ok(cudaMemcpyAsync(hdr, scratch + NOALLOC_MAX_SEGMENTS * 32, 16, cudaMemcpyDeviceToHost, s), "copy status") ||
        !cuda_ok(cudaStreamSynchronize(s), "noalloc segments")) return OMEGA_GPU_FP8GEMM_CHIP_FAIL;
    if (hdr[1] == 1) { set_error("fp8gemm_noalloc: expert ids must be non-decreasing and below the expert count"); return OMEGA_GPU_FP8GEMM_BAD_ARGS; }
    if (hdr[1] == 3) { set_error("fp8gemm_noalloc: a token row index is at or past x_rows (%u)", x_rows); return OMEGA_GPU_FP8GEMM_BAD_ARGS; }
    if (hdr[1] == 2) { set_error("fp8gemm_noalloc: more segments than the fixed table holds"); return OMEGA_GPU_FP8GEMM_TOO_LARGE; }
    GemvArgs a = {};
    a.seg = (const Seg32 *)scratch; a.x = (const void *)(uintptr_t)x_va; a.x_bf16 = x_bf16; a.x_rows = x_rows;
    a.xmap = (const uint32_t *)(uintptr_t)token_rows_va; a.ymap = nullptr;
    a.y = (float *)(uintptr_t)y_va; a.n = t->n; a.k = t->k; a.groups_or_segs = hdr[0]; a.rows = M; a.out_mul = 1.0f;
    return cuda_ok(launch_gemm_rows(a, nullptr, nullptr, s), "fp8gemm_noalloc launch") ? OMEGA_GPU_FP8GEMM_OK : OMEGA_GPU_FP8GEMM_CHIP_FAIL;
}
}  // extern "C"
