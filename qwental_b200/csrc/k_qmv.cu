// Dense batched quantized matvec for GGML IQ3_S (type 21) and Q8_0 (type 8) weights.
//
//   dq_test   decode rows to fp32                      -- role of dq_test, kernels/moe_iq.metal:208-217
//   qmv_gg    fp32 FMA matvec in one fixed order       -- role of qmv_gg,  kernels/qmv_gg.metal:17-39
//   qmv_mma   tensor-core matvec, raw blocks staged by bulk (TMA) copies, one weight pass for up to 64 tokens
//             -- replaces qmv / qmvb / qmv_gg / qmv_ggm for the batched step (src/engine.c:689-769, 5363-5423)
//
// Bind slots follow the reference's qmv_gg (kernels/qmv_gg.metal:18-19): 0 = W, 3 = x (fp16), 4 = y,
// 5 = {N, xstride, ystride, nb} (nb = number of tokens; 0 means the NB define).  Defines: GF (21 | 8),
// KD (K), NB (max tokens), YT_F32 (1: fp32 output, else fp16).
#include "qmv_core.cuh"
#include "qw_kern.h"
#include "tmap.cuh"

using namespace qw;

struct qmv_args {
    uint32_t N, xstride, ystride, nb;
};

// ------------------------------------------------------------------------------------------------ exact decode
// One 32-value segment in the oracle's order: db = d*(1+2*scale), value = +-(db * codebook byte).
template <int GF>
__device__ __forceinline__ void dq32(const uint8_t *row, int sub, float *y, const uint32_t *grid) {
    if (GF == 8) {
        const uint8_t *b = row + (size_t)sub * 34;
        const float d = h2f(ldu16(b));
#pragma unroll
        for (int l = 0; l < 32; l++) y[l] = __fmul_rn(d, (float)(int8_t)b[2 + l]);
        return;
    }
    const uint8_t *b = row + (size_t)(sub >> 3) * 110;
    const int ib = sub & 7;
    const float d = h2f(ldu16(b));
    const uint32_t qh = b[66 + ib];
    const float db = __fmul_rn(d, (float)(1 + 2 * ((b[106 + (ib >> 1)] >> (4 * (ib & 1))) & 15)));
#pragma unroll
    for (int l = 0; l < 4; l++) {
        const uint32_t g1 = __ldg(grid + (b[2 + 8 * ib + 2 * l] | ((qh << (8 - 2 * l)) & 256)));
        const uint32_t g2 = __ldg(grid + (b[2 + 8 * ib + 2 * l + 1] | ((qh << (7 - 2 * l)) & 256)));
        const uint32_t s = b[74 + 4 * ib + l];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float a = __fmul_rn(db, (float)((g1 >> (8 * j)) & 255)), c = __fmul_rn(db, (float)((g2 >> (8 * j)) & 255));
            y[8 * l + j] = (s >> j) & 1 ? -a : a;
            y[8 * l + 4 + j] = (s >> (j + 4)) & 1 ? -c : c;
        }
    }
}

// grid: rows x 32 threads; bytes(2) = {K, row bytes}
template <int GF>
__global__ void dq_test_k(const uint8_t *W, float *y, uint32_t K, uint32_t rb, const uint32_t *grid) {
    pdl_sync();
    const uint32_t r = blockIdx.x, lane = threadIdx.x;
    float v[32];
    for (uint32_t s = lane; s < K / 32; s += 32) {
        dq32<GF>(W + (size_t)r * rb, s, v, grid);
        for (int i = 0; i < 32; i++) y[(size_t)r * K + 32 * s + i] = v[i];
    }
}

static cudaError_t launch_dq_test(const QwLaunch &L) {
    const int gf = (int)L.def("DQ_TEST", L.def("GF", 21));
    struct { uint32_t K, rb; } a = L.bytes<decltype(a)>(2);
    QW_CHECK_ARG(L.buf<uint8_t>(0) && L.buf<float>(1) && a.K % 32 == 0 && L.tx == 32);
    QW_CHECK_ARG((gf == 21 && a.K % 256 == 0) || gf == 8);
    QW_CHECK_ARG(L.avail(0) >= (size_t)L.gx * a.rb && L.avail(1) >= (size_t)L.gx * a.K * 4);
    const uint32_t *grid = ((const QwTables *)L.tables)->grid_u32;
    if (gf == 21) qw_launch(dq_test_k<21>, L.gx, 32, 0, L.stream, L.buf<uint8_t>(0), L.buf<float>(1), a.K, a.rb, grid);
    else qw_launch(dq_test_k<8>, L.gx, 32, 0, L.stream, L.buf<uint8_t>(0), L.buf<float>(1), a.K, a.rb, grid);
    return cudaGetLastError();
}
QW_FAMILY(dq_test, launch_dq_test, 32)

// ------------------------------------------------------------------------------------------------ FMA matvec, canonical order
// One warp per row; lane owns segments lane, lane+32, ...; a segment's 32 products are chained with fma from
// zero and added to the lane accumulator; lanes are reduced by the xor butterfly.  Bit-exact against the CPU
// oracle.  Tokens are processed 8 at a time (the decoded segment is reused for the 8).
template <int GF, bool F32OUT>
__global__ void __launch_bounds__(256) qmv_gg_k(const uint8_t *W, const __half *x, void *y, qmv_args a, uint32_t K, uint32_t rb, const uint32_t *grid) {
    pdl_sync();
    const uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= a.N) return;
    const uint8_t *wr = W + (size_t)row * rb;
    for (uint32_t b0 = 0; b0 < a.nb; b0 += 8) {
        float acc[8];
#pragma unroll
        for (int b = 0; b < 8; b++) acc[b] = 0.f;
        for (uint32_t s = lane; s < K / 32; s += 32) {
            float v[32];
            dq32<GF>(wr, s, v, grid);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                if (b0 + b >= a.nb) continue;
                const uint4 *xp = (const uint4 *)(x + (size_t)(b0 + b) * a.xstride + 32 * s);
                float p = 0.f;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint4 q = __ldcg(xp + i);
                    const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 f = __half22float2(*(const __half2 *)&w4[j]);
                        p = __fmaf_rn(v[8 * i + 2 * j], f.x, p);
                        p = __fmaf_rn(v[8 * i + 2 * j + 1], f.y, p);
                    }
                }
                acc[b] = __fadd_rn(acc[b], p);
            }
        }
#pragma unroll
        for (int b = 0; b < 8; b++) {
            if (b0 + b >= a.nb) continue;
            const float t = warp_sum_canon(acc[b]);
            if (lane == 0) {
                if (F32OUT) ((float *)y)[(size_t)(b0 + b) * a.ystride + row] = t;
                else ((__half *)y)[(size_t)(b0 + b) * a.ystride + row] = __float2half_rn(t);
            }
        }
    }
}

static bool qmv_common_check(const QwLaunch &L, qmv_args &a, int &gf, uint32_t &K, uint32_t &rb, bool &f32) {
    gf = (int)L.def("GF", 21);
    K = (uint32_t)L.def("KD", 0);
    f32 = L.def("YT_F32", 0) != 0;
    a = L.bytes<qmv_args>(5);
    if (a.nb == 0) a.nb = (uint32_t)L.def("NB", 1);
    if (!(gf == 21 || gf == 8) || K == 0 || K % 256 != 0) return false;
    rb = gf == 21 ? K / 256 * 110 : K / 32 * 34;
    if (!L.buf<uint8_t>(0) || !L.buf<__half>(3) || !L.buf<void>(4) || !L.has_bytes(5, 12)) return false;
    if (a.nb == 0 || a.nb > (uint32_t)L.def("ROWS", 64) || a.N == 0 || a.xstride < K || a.xstride % 8 != 0 || a.ystride < a.N) return false;
    if (((uintptr_t)L.buf<__half>(3) & 15) != 0) return false;
    if (L.avail(0) < (size_t)a.N * rb) return false;
    if (L.avail(3) < ((size_t)(a.nb - 1) * a.xstride + K) * 2) return false;
    if (L.avail(4) < ((size_t)(a.nb - 1) * a.ystride + a.N) * (f32 ? 4 : 2)) return false;
    return true;
}

static cudaError_t launch_qmv_gg(const QwLaunch &L) {
    qmv_args a;
    int gf;
    uint32_t K, rb;
    bool f32;
    QW_CHECK_ARG(qmv_common_check(L, a, gf, K, rb, f32));
    QW_CHECK_ARG(L.tx == 256 && L.gx == (a.N + 7) / 8);
    const uint32_t *grid = ((const QwTables *)L.tables)->grid_u32;
    const uint8_t *W = L.buf<uint8_t>(0);
    const __half *x = L.buf<__half>(3);
    void *y = L.buf<void>(4);
#define GO(G, F) qw_launch(qmv_gg_k<G, F>, L.gx, 256, 0, L.stream, W, x, y, a, K, rb, grid)
    if (gf == 21) { if (f32) GO(21, true); else GO(21, false); }
    else { if (f32) GO(8, true); else GO(8, false); }
#undef GO
    return cudaGetLastError();
}
QW_FAMILY(qmv_gg, launch_qmv_gg, 256)

// ------------------------------------------------------------------------------------------------ tensor-core matvec
// Persistent blocks of 8 warps.  An item is a tile of 16*MT rows; the whole tile (full K, rows are contiguous)
// is brought into shared memory by one bulk copy per pipeline stage.  Warp w = (m-tile w / KS, K-slice w % KS)
// walks the units u = ks, ks + KS, ... of its 16 rows; the KS partial tiles of an m-tile are summed in slice
// order 0..KS-1 through shared memory, so the order never depends on the batch.
struct QmvMmaP {
    const uint8_t *W;
    const __half *x;
    void *y;
    const QwTables *tab;
    unsigned *status;
    uint32_t N, K, rb, xstride, ystride, nb, items;
    uint32_t rs;  // qmv_mma2: distance of the rows of a staged tile in shared memory (rb plus padding against bank conflicts)
    // qmv_mma2 with EPX defined: the fp16 output rows are stored into the buffer of every rank (peer memory) and the kernel
    // publishes afterwards -- the all-gather of a projection that every rank runs for its own slots only
    void *yR[8];
    EpPeers ep;  // ep.nranks <= 1: plain local output
};

constexpr int QMV_STAGES = 3;

template <int GF, int NT, int MT, bool F32OUT>
__global__ void __launch_bounds__(256) qmv_mma_k(const QmvMmaP p) {
    constexpr int KS = 8 / MT;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bars = (uint64_t *)smem;                         // QMV_STAGES full barriers
    uint2 *tab = (uint2 *)(smem + 64);                         // 512 x 8 B codebook (IQ3_S only)
    float4 *red = (float4 *)(smem + 64 + 4096);                // [8 warps][NT][32]
    uint8_t *stage0 = smem + 64 + 4096 + 8 * NT * 32 * 16;
    const uint32_t tile_bytes = 16 * MT * p.rb;
    const uint32_t stage_stride = (tile_bytes + 127) & ~127u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int mt = warp / KS, ks = warp % KS;

    if (tid == 0) {
        for (int s = 0; s < QMV_STAGES; s++) mbar_init(&bars[s], 1);
        mbar_init_fence();
    }
    if (GF == 21)
        for (int e = tid; e < 512; e += 256) tab[e] = p.tab->grid_h4[e * 16];
    __syncthreads();

    const uint32_t first = blockIdx.x, step = gridDim.x;
    auto issue = [&](uint32_t j) {  // thread 0 only: item number j of this block into stage j % STAGES
        const uint32_t item = first + j * step;
        if (item >= p.items) return;
        const int s = j % QMV_STAGES;
        mbar_expect_tx(&bars[s], tile_bytes);
        bulk_g2s(stage0 + (size_t)s * stage_stride, p.W + (size_t)item * tile_bytes, tile_bytes, &bars[s]);
    };
    if (tid == 0)
        for (uint32_t j = 0; j < QMV_STAGES - 1; j++) issue(j);

    pdl_sync();  // the weight tiles above do not depend on earlier kernels; the activations and the output do
    // activation rows of this lane's columns
    const uint4 *xcol[NT], *xlo[NT];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        const uint32_t col = g + 8 * nt;
        xcol[nt] = col < p.nb ? (const uint4 *)(p.x + (size_t)col * p.xstride) : nullptr;
        xlo[nt] = nullptr;
    }
    const GridTab<1> gt{tab, 0};
    const uint32_t tile_on = tiles_on<NT>(xcol);
    const int units = p.K / 256;
    bool ok = true;

    for (uint32_t j = 0;; j++) {
        const uint32_t item = first + j * step;
        if (item >= p.items) break;
        if (tid == 0) issue(j + QMV_STAGES - 1);
        const int s = j % QMV_STAGES;
        if (!mbar_wait(&bars[s], (j / QMV_STAGES) & 1)) {
            ok = false;
            break;
        }
        const uint8_t *tile = stage0 + (size_t)s * stage_stride + (size_t)(16 * mt) * p.rb;
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        for (int u = ks; u < units; u += KS)
            unit_mma<GF, NT, 1, false>(tile + (size_t)g * p.rb + (size_t)u * unit_bytes(GF), tile + (size_t)(g + 8) * p.rb + (size_t)u * unit_bytes(GF),
                                       gt, t, xcol, xlo, tile_on, u * 32, acc);
#pragma unroll
        for (int nt = 0; nt < NT; nt++) red[(warp * NT + nt) * 32 + lane] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
        __syncthreads();  // partial tiles visible; every warp is done reading stage s
        // reduce over the KS slices of each m-tile in slice order, then store
        for (int e = tid; e < MT * NT * 32 * 4; e += 256) {
            const int jj = e & 3, ln = (e >> 2) & 31, nt = (e >> 7) % NT, m = (e >> 7) / NT;
            float sum = 0.f;
#pragma unroll
            for (int k2 = 0; k2 < KS; k2++) sum += ((const float *)&red[((m * KS + k2) * NT + nt) * 32 + ln])[jj];
            const uint32_t row = item * 16 * MT + m * 16 + (ln >> 2) + 8 * (jj >> 1);
            const uint32_t col = nt * 8 + 2 * (ln & 3) + (jj & 1);
            if (col < p.nb && row < p.N) {
                if (F32OUT) ((float *)p.y)[(size_t)col * p.ystride + row] = sum;
                else ((__half *)p.y)[(size_t)col * p.ystride + row] = __float2half_rn(sum);
            }
        }
        __syncthreads();  // red may be overwritten, stage s may be refilled
    }
    if (!ok && lane == 0) set_status(p.status, ST_MBAR_TIMEOUT | 1);
}

template <int GF, int NT, int MT, bool F32OUT>
static cudaError_t qmv_mma_go(const QmvMmaP &p, int sm_count, cudaStream_t st) {
    const uint32_t tile_bytes = 16 * MT * p.rb;
    const size_t smem = 64 + 4096 + (size_t)8 * NT * 32 * 16 + (size_t)QMV_STAGES * ((tile_bytes + 127) & ~127u);
    if (smem > 227 * 1024) return cudaErrorInvalidValue;
    auto k = qmv_mma_k<GF, NT, MT, F32OUT>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int occ = 1;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, 256, smem);
    if (e != cudaSuccess) return e;
    if (occ < 1) occ = 1;
    if (occ > 4) occ = 4;
    const uint32_t cap = (uint32_t)(sm_count * occ);
    const uint32_t grid = p.items < cap ? p.items : cap;
    qw_launch(k, grid, 256, smem, st, p);
    return cudaGetLastError();
}

template <int GF, int MT, bool F32OUT>
static cudaError_t qmv_mma_nt(const QmvMmaP &p, int sm, cudaStream_t st) {
    if (p.nb <= 8) return qmv_mma_go<GF, 1, MT, F32OUT>(p, sm, st);
    if (p.nb <= 16) return qmv_mma_go<GF, 2, MT, F32OUT>(p, sm, st);
    if (p.nb <= 32) return qmv_mma_go<GF, 4, MT, F32OUT>(p, sm, st);
    return qmv_mma_go<GF, 8, MT, F32OUT>(p, sm, st);
}

// ---- Variant used for the dense projections: a team of WARPS warps per 16-row tile, one warp per 256-K unit (8 warps
// at K = 2048, 16 at K = 4096); TEAMS teams share one block (and, for IQ3_S, one conflict-free 16-copy codebook of 64 KB
// that arrives by a bulk copy while the activations are loaded).  The activations' B fragments of up to 16 tokens stay
// in registers for the whole kernel.  More than 16 tokens run as passes of 16 over the staged tile (MP): half a unit is decoded into A
// fragments once and all passes run over them, fetching the B fragments per pass.
template <int N>
__device__ __forceinline__ void team_bar(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}
template <int GF, int WARPS, int TEAMS, bool F32OUT, bool MP>
__global__ void __launch_bounds__(WARPS * TEAMS * 32, (WARPS * TEAMS == 8) ? 2 : 1) qmv_mma2_k(const QmvMmaP p) {
    constexpr int NT = 2, TS = 128, STG = GF == 8 ? 2 : QMV_STAGES, UB = GF == 21 ? 110 : 272, TABB = GF == 21 ? 65536 : 0;
    constexpr int TT = WARPS * 32;  // threads of a team
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bars = (uint64_t *)smem;  // [team][STG], then the table's
    uint2 *tab = (uint2 *)(smem + 128);
    const uint32_t tile_bytes = 16 * p.rb, stage_stride = (16 * p.rs + 127) & ~127u;
    const int tid = threadIdx.x, team = tid / TT, tt = tid % TT, warp = tt >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    float4 *red = (float4 *)(smem + 128 + TABB) + team * 2 * WARPS * NT * 32;  // [2][WARPS][NT][32] per team
    uint8_t *stage0 = smem + 128 + TABB + TEAMS * 2 * WARPS * NT * 32 * 16 + (size_t)team * STG * stage_stride;
    uint64_t *full = bars + team * STG;
    pdl_launch();
    if (tid == 0) {
        for (int s = 0; s < TEAMS * STG + 1; s++) mbar_init(&bars[s], 1);
        mbar_init_fence();
        if (GF == 21) {
            mbar_expect_tx(&bars[TEAMS * STG], TABB);
            bulk_g2s(tab, p.tab->grid_h4, TABB, &bars[TEAMS * STG]);
        }
    }
    __syncthreads();
    const uint32_t first = blockIdx.x * TEAMS + team, step = gridDim.x * TEAMS;
    auto issue = [&](uint32_t j) {
        const uint32_t item = first + j * step;
        if (item >= p.items) return;
        const int s = j % STG;
        mbar_expect_tx(&full[s], tile_bytes);
        if (p.rs == p.rb) bulk_g2s(stage0 + (size_t)s * stage_stride, p.W + (size_t)item * tile_bytes, tile_bytes, &full[s]);
        else  // one copy per row, so that the rows land rs bytes apart
            for (uint32_t r = 0; r < 16; r++)
                bulk_g2s(stage0 + (size_t)s * stage_stride + r * p.rs, p.W + (size_t)item * tile_bytes + (size_t)r * p.rb, p.rb, &full[s]);
    };
    if (tt == 0)
        for (uint32_t j = 0; j < STG - 1; j++) issue(j);
    const uint32_t tabc = smem_u32(tab) + (lane & 15) * 8;
    const ZeroRegs zr = zero_regs();
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 xf[NT][8];
    auto load_x = [&]() {  // columns g and 8 + g of this warp's unit
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const uint32_t col = g + 8 * nt;
            const uint4 *xr = (const uint4 *)(p.x + (size_t)col * p.xstride) + warp * 32 + t;
#pragma unroll
            for (int ib = 0; ib < 8; ib++) xf[nt][ib] = col < p.nb ? __ldcg(xr + 4 * ib) : zero;
        }
    };
    pdl_wait();  // weight tiles and the codebook are static; the activations (and the output buffer) are not
    if (!MP) load_x();
    bool ok = GF == 21 ? mbar_wait(&bars[TEAMS * STG], 0) : true;
    const uint32_t passes = (p.nb + 15) / 16;
    uint32_t rb_i = 0;  // alternating reduce buffer
    for (uint32_t j = 0; ok; j++) {
        const uint32_t item = first + j * step;
        if (item >= p.items) break;
        if (tt == 0) issue(j + STG - 1);
        const int s = j % STG;
        if (!mbar_wait(&full[s], (j / STG) & 1)) {
            ok = false;
            break;
        }
        const uint32_t rows = smem_u32(stage0) + s * stage_stride + g * p.rs + warp * UB;
        if constexpr (MP) {
            // more than 16 tokens: decode half a unit once, run every pass of 16 tokens over it (the same MMAs and sums per column)
            float accp[4][NT][4];
#pragma unroll
            for (int ps = 0; ps < 4; ps++)
#pragma unroll
                for (int nt = 0; nt < NT; nt++) accp[ps][nt][0] = accp[ps][nt][1] = accp[ps][nt][2] = accp[ps][nt][3] = 0.f;
            auto run_half = [&](const UnitHalf &A, int hf) {
#pragma unroll
                for (int ps = 0; ps < 4; ps++) {
                    if ((uint32_t)ps >= passes) break;  // warp-uniform
                    const uint32_t ca = ps * 16 + g, cb = ca + 8;
                    const uint4 *xa = (const uint4 *)(p.x + (size_t)ca * p.xstride) + warp * 32 + t + 16 * hf;
                    const uint4 *xb = (const uint4 *)(p.x + (size_t)cb * p.xstride) + warp * 32 + t + 16 * hf;
                    uint4 va[4], vb[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        va[i] = ca < p.nb ? __ldcg(xa + 4 * i) : zero;
                        vb[i] = cb < p.nb ? __ldcg(xb + 4 * i) : zero;
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) half_mma(A, i, zr, va[i], vb[i], (uint32_t)ps * 16 + 8 < p.nb, accp[ps]);
                }
            };
            UnitHalf A;
            if constexpr (GF == 21) {
                const Iq3sHdr h0 = iq3s_hdr(rows, t), h1 = iq3s_hdr(rows + 8 * p.rs, t);
                iq3s_decode_half<0, TS>(rows, rows + 8 * p.rs, t, h0, h1, tabc, A);
                run_half(A, 0);
                iq3s_decode_half<1, TS>(rows, rows + 8 * p.rs, t, h0, h1, tabc, A);
                run_half(A, 1);
            } else {
                q8_decode_half<0>(rows, rows + 8 * p.rs, t, A);
                run_half(A, 0);
                q8_decode_half<1>(rows, rows + 8 * p.rs, t, A);
                run_half(A, 1);
            }
#pragma unroll
            for (int ps = 0; ps < 4; ps++) {
                if ((uint32_t)ps >= passes) break;
                float4 *rd = red + rb_i * WARPS * NT * 32;
                rb_i ^= 1;
#pragma unroll
                for (int nt = 0; nt < NT; nt++) rd[(warp * NT + nt) * 32 + lane] = make_float4(accp[ps][nt][0], accp[ps][nt][1], accp[ps][nt][2], accp[ps][nt][3]);
                team_bar<TT>(team + 1);
                for (int e = tt; e < NT * 32 * 4; e += TT) {
                    const int jj = e & 3, ln = (e >> 2) & 31, nt = e >> 7;
                    float sum = 0.f;
#pragma unroll
                    for (int k2 = 0; k2 < WARPS; k2++) sum += ((const float *)&rd[(k2 * NT + nt) * 32 + ln])[jj];
                    const uint32_t row = item * 16 + (ln >> 2) + 8 * (jj >> 1), col = ps * 16 + nt * 8 + 2 * (ln & 3) + (jj & 1);
                    if (col < p.nb && row < p.N) {
                        if (F32OUT) ((float *)p.y)[(size_t)col * p.ystride + row] = sum;
                        else if (p.ep.nranks > 1) {
                            const __half hv = __float2half_rn(sum);
                            for (uint32_t r = 0; r < p.ep.nranks; r++) ((__half *)p.yR[r])[(size_t)col * p.ystride + row] = hv;
                        } else ((__half *)p.y)[(size_t)col * p.ystride + row] = __float2half_rn(sum);
                    }
                }
            }
        } else
        for (uint32_t ps = 0; ps < passes; ps++) {  // one pass; as a loop it compiles to faster code (four rows, 5120 + 2048 + 151936 outputs: 72.4 against 76.0 us)
            float acc[NT][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            if (GF == 21) unit_mma2<TS>(rows, rows + 8 * p.rs, tabc, t, zr, xf[0], xf[1], ps * 16 + 8 < p.nb, acc);
            else unit_mma2_q8(rows, rows + 8 * p.rs, t, zr, xf[0], xf[1], ps * 16 + 8 < p.nb, acc);
            float4 *rd = red + rb_i * WARPS * NT * 32;
            rb_i ^= 1;
#pragma unroll
            for (int nt = 0; nt < NT; nt++) rd[(warp * NT + nt) * 32 + lane] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
            team_bar<TT>(team + 1);  // partial tiles visible; on the last pass every warp is also done with stage s
            for (int e = tt; e < NT * 32 * 4; e += TT) {
                const int jj = e & 3, ln = (e >> 2) & 31, nt = e >> 7;
                float sum = 0.f;
#pragma unroll
                for (int k2 = 0; k2 < WARPS; k2++) sum += ((const float *)&rd[(k2 * NT + nt) * 32 + ln])[jj];
                const uint32_t row = item * 16 + (ln >> 2) + 8 * (jj >> 1), col = ps * 16 + nt * 8 + 2 * (ln & 3) + (jj & 1);
                if (col < p.nb && row < p.N) {
                    if (F32OUT) ((float *)p.y)[(size_t)col * p.ystride + row] = sum;
                    else if (p.ep.nranks > 1) {
                        const __half hv = __float2half_rn(sum);
                        for (uint32_t r = 0; r < p.ep.nranks; r++) ((__half *)p.yR[r])[(size_t)col * p.ystride + row] = hv;
                    } else ((__half *)p.y)[(size_t)col * p.ystride + row] = __float2half_rn(sum);
                }
            }
        }
    }
    if (!ok && lane == 0) set_status(p.status, ST_MBAR_TIMEOUT | 5);
    if (!F32OUT && p.ep.nranks > 1) ep_publish(p.ep);
}

template <int GF, int WARPS, int TEAMS, bool F32OUT, bool MP = false>
static cudaError_t qmv_mma2_go(const QmvMmaP &p, int sm_count, cudaStream_t st) {
    // more than 16 tokens (at most 64): the form that decodes a unit once for all passes
    if constexpr (!MP) {
        if (p.nb > 16) return qmv_mma2_go<GF, WARPS, TEAMS, F32OUT, true>(p, sm_count, st);
    }
    const size_t smem = 128 + (GF == 21 ? 65536 : 0) + (size_t)TEAMS * 2 * WARPS * 2 * 32 * 16 +
                        (size_t)TEAMS * (GF == 8 ? 2 : QMV_STAGES) * ((16 * p.rs + 127) & ~127u);
    if (smem > 227 * 1024) return cudaErrorInvalidValue;
    auto k = qmv_mma2_k<GF, WARPS, TEAMS, F32OUT, MP>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int occ = 1;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, WARPS * TEAMS * 32, smem);
    if (e != cudaSuccess) return e;
    occ = occ < 1 ? 1 : occ > 4 ? 4 : occ;
    const uint32_t want = (p.items + TEAMS - 1) / TEAMS, cap = (uint32_t)(sm_count * occ), grid = want < cap ? want : cap;
    qw_launch(k, grid, WARPS * TEAMS * 32, smem, st, p);
    return cudaGetLastError();
}

// ---- More than 16 tokens and many rows at K = 2048: a block owns a run of 16-row tiles and walks K in units of 256, so the activations reach a
// block once per round of up to RG tiles instead of once per tile.  (The form above re-reads 256 KB of activations from L2 for each
// 16 rows at 64 tokens: 2.5 GB for an output head of 330 MB -- L2 bandwidth was its bound.)  Two rings feed the block: weights (16-row boxes
// of one Q8_0 unit, or of two IQ3_S units, whose 110 bytes do not start on 16-byte boundaries) and activations (one unit of all tokens,
// 128-byte swizzled).  Warp = (row tile r, token part th): it decodes its tile's unit and runs it against every TS-th column tile.  A
// unit's sum starts from zero and is added to the running total in unit order: the sums of qmv_mma2 in its slice order, bit for bit, without a
// reduction across warps.  MMA column g of a tile holds token (g / 2) + 4 (g % 2), so that the eight lanes of a 16-byte shared load fall into
// eight different chunks of the swizzle.
// TS = warps that share a row tile.  2: the tiles of a block are few (a projection has 3 to 6 per SM) and the warps are what hides
// latency.  1 (Q8_0, 16 tiles per SM and more; IQ3_S by qmv_wide_form): a unit is decoded once for all tokens, by fewer warps with more registers.
// RT = row tiles per warp.  2 (IQ3_S): the activations are read once for both; the weight stages are then one unit long (shared memory).
// Measured on a B200, before -> now, L2 flushed: Q8_0 151936 x 2048, 17 tokens 138 -> 110 us, 61 tokens 253 -> 165 us (TS = 2: 144 and 192);
// IQ3_S 5120 x 2048, 61 tokens 27.2 -> 22.5 us.  330 MB of weights take 50 us.  The head at 61 tokens fills no pipe: shared memory is busy 61 % of the time, the
// tensor pipe 47 %, issue slots 43 %, DRAM 26 % (ncu); with three warps per scheduler a warp issues every 7 cycles, 2.2 of them the latency of its own last
// instruction, 1.9 waiting for loads, 0.8 for the tensor pipe.
template <int GF, int TS, int RT = 1>
struct WideCfg {
    static constexpr int RG = RT * (TS == 2 || GF == 21 ? 7 : 11);  // row tiles per round: 14 + 1 warps of 128 registers, 7 + 1 of up to 255 (with one or two tiles each) or 11 + 1 of 168
    static constexpr int UPW = GF == 21 && RT == 1 ? 2 : 1;             // units per weight stage
    static constexpr int PITCH = GF == 8 ? 272 : UPW == 2 ? 240 : 144;  // bytes between staged rows (eight rows: eight different groups of four banks)
    static constexpr int WS = GF == 21 || TS == 1 ? 2 : 3, XS = 3;  // stages
    static constexpr int TABB = GF == 21 ? 65536 : 0;
    static constexpr int WBYTES = RG * 16 * PITCH;
    static constexpr size_t smem(int CT) { return 1024 + 256 + (size_t)TABB + (size_t)WS * WBYTES + (size_t)XS * CT * TS * 8 * 512; }
};
static_assert(WideCfg<21, 2>::smem(4) <= 227 * 1024 && WideCfg<21, 1>::smem(8) <= 227 * 1024 && WideCfg<21, 1, 2>::smem(8) <= 227 * 1024 && WideCfg<8, 2>::smem(4) <= 227 * 1024 && WideCfg<8, 1>::smem(8) <= 227 * 1024, "shared memory of the wide matvec");

// q8_sub_h for rows 272 bytes apart, in half the shared-memory cycles: 32-bit loads only, and lanes t >= 2 take their words in another
// order, so that rows g and g + 1 do not meet in a bank (only the third load of an even block has two lanes per bank).
template <int IB>
__device__ __forceinline__ float q8_sub_272(uint32_t row, int t, uint32_t (&w)[4]) {
    const bool sw = t >= 2;
    const uint32_t a = row + 8 * t;
    uint32_t lo, hi;
    auto ld = [](uint32_t at) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(at), "n"(34 * IB + (IB & 1 ? 2 : 0)));
        return v;
    };
    if (IB & 1) {
        const uint32_t x1 = ld(a + (sw ? 4 : 0)), x2 = ld(a + (sw ? 0 : 4));
        lo = sw ? x2 : x1;
        hi = sw ? x1 : x2;
    } else {
        const uint32_t x1 = ld(a + (sw ? 4 : 0)), x2 = ld(a + (sw ? 8 : 4)), x3 = ld(a + (sw ? 0 : 8));
        const uint32_t w0 = sw ? x3 : x1, w1 = sw ? x1 : x2, w2 = sw ? x2 : x3;
        lo = __byte_perm(w0, w1, 0x5432);
        hi = __byte_perm(w1, w2, 0x5432);
    }
    q8_pairs(lo, hi, w);
    return h2f((uint16_t)lds_u16<34 * IB>(row));
}

template <int GF, int IB>
__device__ __forceinline__ void wide_decode(uint32_t u0, uint32_t u1, int t, const Iq3sHdr &h0, const Iq3sHdr &h1, uint32_t tabc, uint32_t (&a0)[4],
                                            uint32_t (&a1)[4], float &da, float &db) {
    uint32_t wa[4], wb[4];
    if (GF == 21) {
        da = iq3s_sub_h<IB, 128>(u0 + 2 * t, u0 + t, h0, tabc, wa);
        db = iq3s_sub_h<IB, 128>(u1 + 2 * t, u1 + t, h1, tabc, wb);
    } else {
        da = q8_sub_272<IB>(u0, t, wa);
        db = q8_sub_272<IB>(u1, t, wb);
    }
    a0[0] = wa[0]; a0[1] = wb[0]; a0[2] = wa[1]; a0[3] = wb[1];
    a1[0] = wa[2]; a1[1] = wb[2]; a1[2] = wa[3]; a1[3] = wb[3];
}

// CT = column tiles of 8 tokens per warp: up to 8 CT TS tokens per block; more tokens (a piece of a prompt) are groups of 64 that share
// the grid: blocks_per_group blocks each, so that a group's blocks have many row tiles and run them side by side.  One launch for all groups
// instead of one per 64 tokens, and K = 4096 here instead of in qmv_mma2: a prompt of 419 tokens, 48 layers, 42.5 -> 39.6 ms, 1700 tokens, 12
// layers, 41.2 -> 38.9 ms on a B200.  UNITS = K / 256.  grid: at most one block per SM
template <int GF, bool F32OUT, int TS, int CT, int UNITS, int RT = 1>
__global__ void __launch_bounds__((TS * WideCfg<GF, TS, RT>::RG / RT + 1) * 32, 1) qmv_wide_k(const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mx,
                                                                                    const QmvMmaP p, uint32_t rg, uint32_t blocks_per_group) {
    using C = WideCfg<GF, TS, RT>;
    constexpr int WS = C::WS, XS = C::XS, UPW = C::UPW, R = 8 * CT * TS, XBYTES = R * 512, CH = CT <= 4 ? CT : CT / 2;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023) & ~1023u;  // the swizzle pattern repeats every 1024 bytes
    const uint32_t xs0 = base, ws0 = xs0 + XS * XBYTES, tab0 = ws0 + WS * C::WBYTES;
    uint64_t *bars = (uint64_t *)(smem_raw + (tab0 + C::TABB - smem_u32(smem_raw)));
    uint64_t *wfull = bars, *wempty = wfull + WS, *xfull = wempty + WS, *xempty = xfull + XS, *tbar = xempty + XS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const uint32_t ncw = TS * rg / RT;  // consumer warps; warp ncw is the producer
    pdl_launch();
    if (tid == 0) {
        for (int s = 0; s < WS; s++) { mbar_init(&wfull[s], 1); mbar_init(&wempty[s], ncw); }
        for (int s = 0; s < XS; s++) { mbar_init(&xfull[s], 1); mbar_init(&xempty[s], ncw); }
        mbar_init(tbar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    // this block's tiles, and the tiles of a round: both split evenly
    const uint32_t c0 = blockIdx.x / blocks_per_group * 64, bi = blockIdx.x % blocks_per_group;  // first token of the group, block within it
    const uint32_t t0 = (uint32_t)((uint64_t)bi * p.items / blocks_per_group), cnt = (uint32_t)((uint64_t)(bi + 1) * p.items / blocks_per_group) - t0;
    const uint32_t rounds = (cnt + rg - 1) / rg;
    if ((uint32_t)warp == ncw) {
        if (lane == 0) {
            bool ok = true;
            if (GF == 21) {
                mbar_expect_tx(tbar, C::TABB);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(tab0), "l"(p.tab->grid_h4), "r"(C::TABB),
                             "r"(smem_u32(tbar))
                             : "memory");
            }
            const uint32_t nw = rounds * (UNITS / UPW), nx = rounds * UNITS;
            uint32_t jw = 0;
            auto put_w = [&]() {  // weight stage number jw
                const uint32_t s = jw % WS, r = jw / (UNITS / UPW), kp = jw % (UNITS / UPW);
                if (jw >= WS && !mbar_wait(&wempty[s], (jw / WS - 1) & 1)) return false;
                const uint32_t lo = cnt * r / rounds, n = cnt * (r + 1) / rounds - lo;
                mbar_expect_tx(&wfull[s], n * 16 * C::PITCH);
                const int xc = GF == 21 ? (int)((110 * UPW * kp) & ~15u) : (int)(136 * kp);  // bytes, or pairs of bytes
                for (uint32_t i = 0; i < n; i++) tma_load_2d(ws0 + s * C::WBYTES + i * 16 * C::PITCH, &mw, xc, (int)((t0 + lo + i) * 16), &wfull[s]);
                jw++;
                return true;
            };
            while (jw < WS && jw < nw) put_w();  // the first weights do not depend on earlier kernels; the activations and the output do
            pdl_wait();
            for (uint32_t jx = 0; jx < nx && ok; jx++) {
                const uint32_t s = jx % XS, u = jx % UNITS;
                if (jx >= XS && !mbar_wait(&xempty[s], (jx / XS - 1) & 1)) { ok = false; break; }
                mbar_expect_tx(&xfull[s], XBYTES);
                for (uint32_t q = 0; q < 4; q++) tma_load_2d(xs0 + s * XBYTES + q * R * 128, &mx, (int)(u * 256 + q * 64), (int)c0, &xfull[s]);
                // weights as far ahead as their ring allows without holding up the activations of the stages already in it
                if (jw < nw && jw * UPW <= jx + (WS - 1) * UPW) ok = put_w();
            }
            if (!ok) set_status(p.status, ST_MBAR_TIMEOUT | 12);
        }
        return;
    }
    pdl_wait();
    const uint32_t r = (uint32_t)warp % (rg / RT) * RT, th = (uint32_t)warp / (rg / RT);
    // (this warp's column tiles: th, th + TS, ...; rows past the last token read as zero)
    const uint32_t tokr = (uint32_t)(g >> 1) | ((uint32_t)(g & 1) << 2);                      // token of MMA column g within a tile
    const uint32_t xoff = th * 1024 + tokr * 128 + ((uint32_t)t ^ tokr) * 16, tabc = tab0 + (lane & 15) * 8;
    const ZeroRegs zr = zero_regs();
    bool ok = GF == 21 ? mbar_wait(tbar, 0) : true;
    uint32_t jw = 0, jx = 0;
    for (uint32_t rd = 0; rd < rounds && ok; rd++) {
        const uint32_t lo = cnt * rd / rounds, n = cnt * (rd + 1) / rounds - lo;
        float tot[RT][CT][4];
#pragma unroll
        for (int i = 0; i < RT * CT; i++) tot[i / CT][i % CT][0] = tot[i / CT][i % CT][1] = tot[i / CT][i % CT][2] = tot[i / CT][i % CT][3] = 0.f;
#pragma unroll 1
        for (uint32_t u = 0; u < UNITS; u++, jx++) {
            if (u % UPW == 0 && !mbar_wait(&wfull[jw % WS], (jw / WS) & 1)) { ok = false; break; }
            if (!mbar_wait(&xfull[jx % XS], (jx / XS) & 1)) { ok = false; break; }
            if (r < n) {  // (a second row tile past the round's last one is computed from whatever the stage holds, and not stored)
                const uint32_t u0 = ws0 + (jw % WS) * C::WBYTES + (r * 16 + g) * C::PITCH + (GF == 21 ? ((110 * UPW * (u / UPW)) & 15) + (u % UPW) * 110 : 0);
                const uint32_t u1 = u0 + 8 * C::PITCH, xa = xs0 + (jx % XS) * XBYTES + xoff;
                Iq3sHdr h0[RT]{}, h1[RT]{};
                float acc[RT][CT][4];
#pragma unroll
                for (int i = 0; i < RT * CT; i++) acc[i / CT][i % CT][0] = acc[i / CT][i % CT][1] = acc[i / CT][i % CT][2] = acc[i / CT][i % CT][3] = 0.f;
                // The MMAs of the column tiles are issued back to back, first halves then second halves, and the next sub-block is decoded before
                // their results are used: in program order one tile after the other, every tile waited for its load and for two dependent MMAs.
                uint32_t a0[RT][4], a1[RT][4];
                float da[RT], db[RT];
#pragma unroll
                for (int m = 0; m < RT; m++) {
                    if (GF == 21) {
                        h0[m] = iq3s_hdr(u0 + m * 16 * C::PITCH, t);
                        h1[m] = iq3s_hdr(u1 + m * 16 * C::PITCH, t);
                    }
                    wide_decode<GF, 0>(u0 + m * 16 * C::PITCH, u1 + m * 16 * C::PITCH, t, h0[m], h1[m], tabc, a0[m], a1[m], da[m], db[m]);
                }
#define WIDE_SUB(IB)                                                                                                              \
    {                                                                                                                             \
        const uint32_t xb = (IB & 1 ? xa ^ 64u : xa) + (IB / 2) * R * 128;                                                        \
        float ea[RT], eb[RT];                                                                                                     \
        _Pragma("unroll") for (int m = 0; m < RT; m++) {                                                                          \
            ea[m] = da[m];                                                                                                        \
            eb[m] = db[m];                                                                                                        \
        }                                                                                                                         \
        _Pragma("unroll") for (int c = 0; c < CT; c += CH) { /* CH column tiles at a time: registers */                           \
            uint4 xv[CH];                                                                                                         \
            _Pragma("unroll") for (int i = 0; i < CH; i++) xv[i] = lds_v4(xb + (c + i) * TS * 1024);                              \
            _Pragma("unroll") for (int m = 0; m < RT; m++) {                                                                      \
                float q[CH][4];                                                                                                   \
                _Pragma("unroll") for (int i = 0; i < CH; i++) mma_f16(q[i], a0[m], xv[i].x, xv[i].y, zr.z);                      \
                _Pragma("unroll") for (int i = 0; i < CH; i++) mma_f16(q[i], a1[m], xv[i].z, xv[i].w, q[i]);                      \
                if (IB < 7 && c + CH == CT)                                                                                       \
                    wide_decode<GF, (IB < 7 ? IB + 1 : 7)>(u0 + m * 16 * C::PITCH, u1 + m * 16 * C::PITCH, t, h0[m], h1[m], tabc, a0[m], a1[m], da[m], db[m]); \
                _Pragma("unroll") for (int i = 0; i < CH; i++) {                                                                  \
                    acc[m][c + i][0] = fmaf(ea[m], q[i][0], acc[m][c + i][0]);                                                    \
                    acc[m][c + i][1] = fmaf(ea[m], q[i][1], acc[m][c + i][1]);                                                    \
                    acc[m][c + i][2] = fmaf(eb[m], q[i][2], acc[m][c + i][2]);                                                    \
                    acc[m][c + i][3] = fmaf(eb[m], q[i][3], acc[m][c + i][3]);                                                    \
                }                                                                                                                 \
            }                                                                                                                     \
        }                                                                                                                         \
    }
                WIDE_SUB(0) WIDE_SUB(1) WIDE_SUB(2) WIDE_SUB(3) WIDE_SUB(4) WIDE_SUB(5) WIDE_SUB(6) WIDE_SUB(7)
#undef WIDE_SUB
#pragma unroll
                for (int i = 0; i < RT * CT; i++)
#pragma unroll
                    for (int k = 0; k < 4; k++) tot[i / CT][i % CT][k] += acc[i / CT][i % CT][k];
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&xempty[jx % XS]);
                if (u % UPW == UPW - 1) mbar_arrive(&wempty[jw % WS]);
            }
            if (u % UPW == UPW - 1) jw++;
        }
        if (!ok || r >= n) continue;
#pragma unroll
        for (int m = 0; m < RT; m++) {
            if (RT > 1 && r + m >= n) break;
            const uint32_t row = (t0 + lo + r + m) * 16 + g;
#pragma unroll
            for (int i = 0; i < CT; i++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t col = c0 + (TS * i + th) * 8 + t + 4 * (k & 1), rw = row + 8 * (k >> 1);
                    if (col >= p.nb) continue;
                    if (F32OUT) ((float *)p.y)[(size_t)col * p.ystride + rw] = tot[m][i][k];
                    else ((__half *)p.y)[(size_t)col * p.ystride + rw] = __float2half_rn(tot[m][i][k]);
                }
        }
    }
    if (!ok && lane == 0) set_status(p.status, ST_MBAR_TIMEOUT | 13);
}

template <int GF, bool F32OUT, int TS, int UNITS, int RT = 1>
static cudaError_t qmv_wide_ts(const QmvMmaP &p, uint32_t groups, uint32_t bpg, uint32_t per, cudaStream_t st) {
    using C = WideCfg<GF, TS, RT>;
    CUtensorMap mw, mx;
    constexpr int B = 2 / TS;  // column tiles per 16 tokens of a warp
    const int n = p.nb <= 32 ? 2 : p.nb <= 48 ? 3 : 4, ct = n * B;
    const bool mok = GF == 21 ? tmap_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.W, p.rb, p.N, p.rb, C::PITCH, 16, CU_TENSOR_MAP_SWIZZLE_NONE)
                              : tmap_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT16, p.W, p.rb / 2, p.N, p.rb, 136, 16, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (!mok || !tmap_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, p.x, p.K, p.nb, (uint64_t)p.xstride * 2, 64, 16 * n, CU_TENSOR_MAP_SWIZZLE_128B))
        return cudaErrorInvalidValue;
    auto k = n == 2 ? qmv_wide_k<GF, F32OUT, TS, 2 * B, UNITS, RT> : n == 3 ? qmv_wide_k<GF, F32OUT, TS, 3 * B, UNITS, RT> : qmv_wide_k<GF, F32OUT, TS, 4 * B, UNITS, RT>;
    const size_t smem = C::smem(ct);
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // as many row tiles per round as split the block's tiles into equal rounds of at most RG
    const uint32_t rounds = (per + C::RG - 1) / C::RG, rg = ((per + rounds - 1) / rounds + RT - 1) / RT * RT;
    qw_launch(k, groups * bpg, (TS * rg / RT + 1) * 32, smem, st, mw, mx, p, rg, bpg);
    return cudaGetLastError();
}
// IQ3_S, more than 64 tokens: two warps per row tile (0), one (1), or one per pair of row tiles (2)?  What a block's `per` row tiles cost in each is rounds times the time of
// a round, and that goes by the busiest of the SM's four schedulers: decode and MMAs of half the tokens of a tile, of a tile, or of two.  Tables: times of a round of 1 to 7 tiles
// (0, 1; a warp idle in a shorter round frees no other scheduler), of up to 8 and of up to 14 tiles (2), in half microseconds at K = 2048.  Measured on a B200 (L2
// flushed) with 1 to 32 tiles per block, 2 to 16 groups of 64 tokens, K = 2048 and 4096: the ratios depend on the tiles alone.  Time of 0 at K = 2048, us; ratios of 1 and 2 to it:
//   tiles  0    1    2         tiles  0    1    2         tiles  0    1    2          tiles  0    1    2
//     1   18  1.11 1.68         6    26  1.03 1.17         14   50  0.94 0.87          21   72  0.91 1.05
//     3   22  1.01 1.40         7    30  0.95 1.10         15   59  1.08 0.96          24   79  1.06 0.97
//     4   22  0.96 1.33         8    36  0.96 0.93         16   60  1.06 0.95          28   93  0.91 0.85
//     5   26  1.06 1.20        12    44  1.05 0.99         18   61  1.06 1.23          30   95  1.07 1.16
// With 1 for three and more groups, and 2 where the rounds nearly halve, whatever the tiles: 12352 x 2048, 129 to 192 tokens, 66 us, now 58 to 60; 9216 x 2048, 193 to
// 256, 66 -> 60; 5120 x 2048, 385 to 448, 64 -> 57; 4800 x 4096, 385 to 448, 116 -> 102.  Prompts of 160, 192 and 1024 tokens, 12 layers: 4.30 -> 4.22, 4.51 -> 4.40 and 13.47 -> 13.32 ms.
static int qmv_wide_form(uint32_t per) {
    constexpr uint32_t T0[7] = {19, 20, 26, 27, 33, 34, 42}, T1[7] = {22, 23, 25, 25, 37, 37, 38};
    const uint32_t r7 = (per + 6) / 7, t7 = (per + r7 - 1) / r7, r14 = (per + 13) / 14, t14 = (per + r14 - 1) / r14;
    const uint32_t c0 = r7 * T0[t7 - 1], c1 = r7 * T1[t7 - 1], c2 = r14 * (t14 <= 8 ? 49 : 68);
    return c2 <= c0 && c2 <= c1 ? 2 : c1 < c0 ? 1 : 0;
}
template <int GF, bool F32OUT, int UNITS = 8>
static cudaError_t qmv_wide_go(const QmvMmaP &p, int sm_count, cudaStream_t st) {
    // one block per SM, shared evenly by the groups of 64 tokens
    const uint32_t groups = (p.nb + 63) / 64, most = (uint32_t)sm_count / groups > 0 ? (uint32_t)sm_count / groups : 1, bpg = p.items < most ? p.items : most;
    const uint32_t per = (p.items + bpg - 1) / bpg;
    const int form = GF == 8 ? per >= 16 : groups > 1 ? qmv_wide_form(per) : 0;
    if constexpr (GF == 21)
        if (form == 2) return qmv_wide_ts<GF, F32OUT, 1, UNITS, 2>(p, groups, bpg, per, st);
    if (form == 1) return qmv_wide_ts<GF, F32OUT, 1, UNITS>(p, groups, bpg, per, st);
    return qmv_wide_ts<GF, F32OUT, 2, UNITS>(p, groups, bpg, per, st);
}

// More than 16 tokens at K = 2048: the wide form, or the one that decodes a unit once for all passes of 16 tokens (qmv_mma2 with MP)?  A
// block of the wide form walks K alone and costs the same for one row tile as for a few, and its copies and barriers come first; MP splits
// K over 8 warps, but reads the activations once per tile: the more tokens, the fewer tiles make up for it.  Time of MP over time of wide on a
// B200, 148 SMs, IQ3_S / Q8_0:
//   row tiles        17 tokens     24 tokens     32 tokens     41 tokens     48 tokens     64 tokens
//    16             0.85 / 0.69   0.85 / 0.69   0.88 / 0.72   0.84 / 0.77   0.87 / 0.77   0.86 / 0.69
//   128             0.83 / 0.83   0.85 / 0.86   0.89 / 0.89   0.88 / 0.97   0.93 / 1.00   0.92 / 0.89
//   185             0.79 / 0.75   0.85 / 0.76   0.92 / 0.85   0.96 / 1.00   1.05 / 1.12   1.10 / 1.09
//   296             0.81 / 0.78   0.85 / 0.83   0.92 / 0.88   0.99 / 1.05   1.09 / 1.16   1.13 / 1.15
//   370             1.02 / 0.93   1.05 / 1.05   1.11 / 1.15   1.19 / 1.25   1.27 / 1.34   1.31 / 1.34
//   592             0.96 / 0.97   1.02 / 1.05   1.10 / 1.13   1.24 / 1.33   1.36 / 1.47   1.44 / 1.49
//   772             1.02 / 1.02   1.05 / 1.10   1.14 / 1.21   1.31 / 1.39   1.41 / 1.50   1.52 / 1.57
// So: wide beyond 4, 2 or 1 row tiles per SM (up to 21, up to 42, more tokens).  One more tile than that costs MP little, a last round for few
// teams, and wide a whole round (297 tiles: 0.85 to 1.05): an eighth is added.
static bool qmv_wide_pays(uint32_t items, uint32_t nb, uint32_t sms) {
    const uint32_t per_sm = nb <= 21 ? 4 : nb <= 42 ? 2 : 1;
    return 8 * items > (8 * per_sm + 1) * sms;
}

// The grid and block given by the host are ignored (the kernels are persistent and size themselves).  Defines: GF (21 = IQ3_S,
// 8 = Q8_0), KD, YT_F32; EPX = ranks of a slot-sharded projection whose rows go to every rank (see below).
static cudaError_t launch_qmv_mma(const QwLaunch &L) {
    qmv_args a;
    int gf;
    uint32_t K, rb;
    bool f32;
    QW_CHECK_ARG(qmv_common_check(L, a, gf, K, rb, f32));
    QW_CHECK_ARG(L.tx == 256 || L.tx == 512);
    // rows per item: fixed by the matrix shape alone (never by the batch), so results do not depend on nb
    const int mt = 1;
    QW_CHECK_ARG(a.N % (16 * mt) == 0 && ((uintptr_t)L.buf<uint8_t>(0) & 15) == 0 && (16 * rb) % 16 == 0);
    QmvMmaP p{};
    p.W = L.buf<uint8_t>(0);
    p.x = L.buf<__half>(3);
    p.y = L.buf<void>(4);
    p.tab = (const QwTables *)L.tables;
    p.status = L.status;
    p.N = a.N; p.K = K; p.rb = rb; p.xstride = a.xstride; p.ystride = a.ystride; p.nb = a.nb;
    p.items = a.N / (16 * mt);
    // Rows of a staged tile: the eight rows a warp instruction touches must fall into different banks.  An IQ3_S lane
    // reads 2 bytes (row distance = 4, 12, 20 or 28 words mod 32), a Q8_0 lane 8 bytes (8 or 24 words mod 32: two rows
    // per bank group, the best a 32-byte-per-row access allows).  Padding is a multiple of 16 bytes (bulk-copy alignment).
    p.rs = rb;
    for (uint32_t pad = 0; pad < 128 && rb % 16 == 0; pad += 16) {
        const uint32_t wds = ((rb + pad) / 4) % 32;
        if (gf == 21 ? (wds % 8 == 4) : (wds % 16 == 8)) {
            p.rs = rb + pad;
            break;
        }
    }
    const uint32_t epx = (uint32_t)L.def("EPX", 0);
    if (epx > 1) {
        // binds 16 + r = y of rank r (row 0 = this rank's first row, as bind 4), 24 + r = flag array of rank r,
        // 11 = {seq, done} counters, 12 = {rank}; only for the fp16-output IQ3_S projections of the persistent kernel
        QW_CHECK_ARG(epx <= 8 && !f32 && gf == 21 && (K == 2048 || K == 4096) && L.has_bytes(12, 4) && L.buf<unsigned>(11) && L.avail(11) >= 8);
        p.ep.nranks = epx;
        p.ep.rank = L.bytes<uint32_t>(12);
        QW_CHECK_ARG(p.ep.rank < epx);
        p.ep.seq = L.buf<unsigned>(11);
        p.ep.done = p.ep.seq + 1;
        for (uint32_t r = 0; r < epx; r++) {
            p.yR[r] = L.buf<void>(16 + r);
            p.ep.flagR[r] = L.buf<unsigned>(24 + r);
            QW_CHECK_ARG(p.yR[r] && p.ep.flagR[r] && L.avail(24 + r) >= epx * 4 && L.avail(16 + r) >= ((size_t)(a.nb - 1) * a.ystride + a.N) * 2);
        }
    }
#define GO(G, M)                                                        \
    return f32 ? qmv_mma_nt<G, M, true>(p, L.sm_count, L.stream) : qmv_mma_nt<G, M, false>(p, L.sm_count, L.stream)
    // More than 16 tokens: the activations no longer fit a warp's registers, and the wide form reads them from shared memory.  (The
    // exchange between ranks is built into qmv_mma2 only, more than 64 tokens into the wide form.)
    if (K == 2048 && a.nb > 16 && epx <= 1 && (a.nb > 64 || qmv_wide_pays(p.items, a.nb, (uint32_t)L.sm_count))) {
        if (gf == 21) return f32 ? qmv_wide_go<21, true>(p, L.sm_count, L.stream) : qmv_wide_go<21, false>(p, L.sm_count, L.stream);
        return f32 ? qmv_wide_go<8, true>(p, L.sm_count, L.stream) : qmv_wide_go<8, false>(p, L.sm_count, L.stream);
    }
    // More than 64 tokens (ROWS defined: a piece of a prompt) at K = 4096 too: with 64 a block would have one row tile, with several groups of
    // tokens it has enough to keep its warps busy.
    if (a.nb > 64) {
        QW_CHECK_ARG(gf == 21 && K == 4096 && epx <= 1);
        return f32 ? qmv_wide_go<21, true, 16>(p, L.sm_count, L.stream) : qmv_wide_go<21, false, 16>(p, L.sm_count, L.stream);
    }
    if (gf == 21 && K == 2048) return f32 ? qmv_mma2_go<21, 8, 2, true>(p, L.sm_count, L.stream) : qmv_mma2_go<21, 8, 2, false>(p, L.sm_count, L.stream);
    if (gf == 21 && K == 4096) return f32 ? qmv_mma2_go<21, 16, 1, true>(p, L.sm_count, L.stream) : qmv_mma2_go<21, 16, 1, false>(p, L.sm_count, L.stream);
    if (gf == 8 && K == 2048) return f32 ? qmv_mma2_go<8, 8, 1, true>(p, L.sm_count, L.stream) : qmv_mma2_go<8, 8, 1, false>(p, L.sm_count, L.stream);
    if (gf == 21) GO(21, 1);
    else GO(8, 1);
#undef GO
}
QW_FAMILY(qmv_mma, launch_qmv_mma, 256)
