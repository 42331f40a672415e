// Ragged paged-KV gated GQA decode attention for all slots in one launch: split-K over the slot's pages with a
// log-sum-exp merge.
//
//   qsa_prep   per head: RMSNorm(q)*w, partial RoPE (first 64 dims, pairs (i, i+32), theta 1e7), write q;
//              RMSNorm(k)*w + RoPE -> K page, v -> V page at the slot's position
//              -- role of qsa_prep_f, kernels/qsa_dec.metal:68-127 (dense part: no indexer)
//   qsa_attn   one block per (page chunk, kv head, slot): online softmax over the chunk's tokens for the
//              GQA = QH/KVH query heads of that kv head, partial (acc, m, l) out
//              -- role of qsa_attn5 (dense branch), kernels/qsa_dec.metal:481-600
//   qsa_merge  log-sum-exp merge of a slot's partials in chunk order, y = fp16(fp16(o/L) * sigmoid(gate));
//              gate = second half of each head's q-projection output
//              -- role of qsa_merge4, kernels/qsa_dec.metal:609-645
//
// KV layout (new; the reference keeps one contiguous buffer per slot, src/engine.c:857-930): a pool of pages of
// 256 tokens; page p, attention layer l holds K [KVH][256][HD] then V [KVH][256][HD] in fp16, so one kv head's
// 256 keys are one contiguous 128 KB run.  A slot owns a list of page ids (its page table row).
// The reference launches the core once per slot (src/engine.c:8948-8959); here slot and chunk are grid
// dimensions, chunks past a slot's length exit at once, and the chunking of a slot depends only on its own
// length, so a slot's result is bit-identical alone or in any batch.
#include "common.cuh"
#include "qw_kern.h"
#include "tmap.cuh"
#include <cstdio>
#include <map>
#include <mutex>

using namespace qw;

#define QSA_EPS 1e-6f
#define QSA_PAGE 256

struct qsa_args {
    uint32_t nb, layer, nlayers, qkv_stride;  // qkv row: [QH x (q HD | gate HD)] [KVH x k HD] [KVH x v HD]
    uint32_t max_pages, max_chunks, pad0, pad1;
};

__device__ __forceinline__ size_t page_base(uint32_t page, uint32_t layer, uint32_t nlayers, uint32_t KVH, uint32_t HD) {
    return ((size_t)page * nlayers + layer) * 2 * KVH * QSA_PAGE * HD;  // in halves
}

// binds: 0 = qkv fp16 [nb][qkv_stride], 1 = q norm w fp32 [HD], 2 = k norm w fp32 [HD], 3 = q out fp16 [nb][QH][HD],
// 4 = KV pool fp16, 5 = page table int32 [slots][max_pages], 6 = pos int32 [nb] (tokens already in the cache),
// 7 = slot ids int32 [nb], 8 = qsa_args.   grid (QH + KVH, nb) x 256 (HD = 256)
__global__ void __launch_bounds__(256) qsa_prep_k(const __half *qkv, const float *qn, const float *kn, __half *q, __half *pool, const int32_t *pt,
                                                  const int32_t *posv, const int32_t *sids, qsa_args a, uint32_t QH, uint32_t KVH) {
    constexpr uint32_t HD = 256, RD = 64;
    __shared__ float tmp[8], v[HD];
    pdl_sync();
    const uint32_t hh = blockIdx.x, t = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t pos = (uint32_t)posv[t];
    const bool isq = hh < QH;
    const uint32_t kh = hh - QH;
    const __half *row = qkv + (size_t)t * a.qkv_stride;
    const float x = isq ? __half2float(row[hh * 2 * HD + tid]) : __half2float(row[QH * 2 * HD + kh * HD + tid]);
    const float p = warp_sum(x * x);
    if (lane == 0) tmp[warp] = p;
    __syncthreads();
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) ss += tmp[i];
    const float r = rsqrtf(ss / HD + QSA_EPS);
    v[tid] = x * r * (isq ? qn[tid] : kn[tid]);
    __syncthreads();
    if (tid < RD / 2) {
        const float f = powf(10000000.0f, -(float)(2 * tid) / (float)RD) * (float)pos;
        const float c = cosf(f), s = sinf(f);
        const float x1 = v[tid], x2 = v[tid + RD / 2];
        v[tid] = x1 * c - x2 * s;
        v[tid + RD / 2] = x2 * c + x1 * s;
    }
    __syncthreads();
    if (isq) {
        q[((size_t)t * QH + hh) * HD + tid] = __float2half_rn(v[tid]);
    } else {
        const uint32_t page = (uint32_t)pt[(size_t)sids[t] * a.max_pages + pos / QSA_PAGE];
        __half *pb = pool + page_base(page, a.layer, a.nlayers, KVH, HD);
        const size_t o = ((size_t)kh * QSA_PAGE + pos % QSA_PAGE) * HD + tid;
        pb[o] = __float2half_rn(v[tid]);
        pb[(size_t)KVH * QSA_PAGE * HD + o] = row[QH * 2 * HD + KVH * HD + kh * HD + tid];
    }
}

static bool qsa_dims(const QwLaunch &L, uint32_t &QH, uint32_t &KVH, uint32_t &HD) {
    QH = (uint32_t)L.def("QH", 16);
    KVH = (uint32_t)L.def("KVH", 2);
    HD = (uint32_t)L.def("HD", 256);
    return HD == 256 && QH % KVH == 0 && QH / KVH == 8;
}

static cudaError_t launch_qsa_prep(const QwLaunch &L) {
    uint32_t QH, KVH, HD;
    QW_CHECK_ARG(qsa_dims(L, QH, KVH, HD));
    qsa_args a = L.bytes<qsa_args>(8);
    QW_CHECK_ARG(L.has_bytes(8, 24) && a.nb >= 1 && a.nb <= (uint32_t)L.def("ROWS", 64) && a.layer < a.nlayers && a.qkv_stride >= QH * 2 * HD + 2 * KVH * HD);
    for (int i = 0; i <= 7; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= ((size_t)(a.nb - 1) * a.qkv_stride + QH * 2 * HD + 2 * KVH * HD) * 2 && L.avail(3) >= (size_t)a.nb * QH * HD * 2 &&
                 L.avail(6) >= (size_t)a.nb * 4 && L.avail(7) >= (size_t)a.nb * 4 && L.tx == 256);
    qw_launch(qsa_prep_k, dim3(QH + KVH, a.nb), 256, 0, L.stream, L.buf<__half>(0), L.buf<float>(1), L.buf<float>(2), L.buf<__half>(3), L.buf<__half>(4),
                                                          L.buf<int32_t>(5), L.buf<int32_t>(6), L.buf<int32_t>(7), a, QH, KVH);
    return cudaGetLastError();
}
QW_FAMILY(qsa_prep, launch_qsa_prep, 256)

// ------------------------------------------------------------------------------------------------ attention core
// Chunk = one page (256 tokens).  Block = 8 warps = the 8 query heads of one kv head; lane owns 8 of the 256
// dims; 4 tokens per iteration (scores by warp reduction, then the online-softmax update), the expression of
// kernels/qsa_dec.metal:520-539.  part [nb][max_chunks][QH][HD + 2] fp32 (acc, m, l).
// binds: 0 = q fp16 [nb][QH][HD], 1 = KV pool, 2 = page table, 3 = pos (tokens in the cache before this step;
// the step's own token was appended by qsa_prep, so the slot attends to pos + 1 tokens), 4 = slot ids,
// 5 = part, 6 = qsa_args.   grid (max_chunks, KVH, nb) x 256
__global__ void __launch_bounds__(256) qsa_attn_k(const __half *q, const __half *pool, const int32_t *pt, const int32_t *posv, const int32_t *sids,
                                                  float *part, qsa_args a, uint32_t QH, uint32_t KVH) {
    constexpr uint32_t HD = 256, PL = 8, U4 = 4;
    pdl_sync();
    const uint32_t ch = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
    const uint32_t ntok = (uint32_t)posv[t] + 1;
    if (ch * QSA_PAGE >= ntok) return;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qh = kvh * 8 + warp;
    const uint32_t n = min((uint32_t)QSA_PAGE, ntok - ch * QSA_PAGE);
    const uint32_t page = (uint32_t)pt[(size_t)sids[t] * a.max_pages + ch];
    const __half *Kp = pool + page_base(page, a.layer, a.nlayers, KVH, HD) + (size_t)kvh * QSA_PAGE * HD + lane * PL;
    const __half *Vp = Kp + (size_t)KVH * QSA_PAGE * HD;
    const float scale = rsqrtf((float)HD);
    float qv[PL], acc[PL];
    {
        const uint4 qq = *(const uint4 *)(q + ((size_t)t * QH + qh) * HD + lane * PL);
        const uint32_t w4[4] = {qq.x, qq.y, qq.z, qq.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(*(const __half2 *)&w4[j]);
            qv[2 * j] = f.x * scale;
            qv[2 * j + 1] = f.y * scale;
        }
    }
#pragma unroll
    for (int d = 0; d < PL; d++) acc[d] = 0.f;
    float m = -INFINITY, l = 0.f;
    for (uint32_t i = 0; i < n; i += U4) {
        float s[U4];
        uint4 vv[U4];
#pragma unroll
        for (uint32_t u = 0; u < U4; u++) {
            const bool ok = i + u < n;
            const uint32_t tk = ok ? i + u : i;
            const uint4 kk = __ldcg((const uint4 *)(Kp + (size_t)tk * HD));
            vv[u] = __ldcg((const uint4 *)(Vp + (size_t)tk * HD));
            const uint32_t w4[4] = {kk.x, kk.y, kk.z, kk.w};
            float d = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(*(const __half2 *)&w4[j]);
                d = fmaf(f.x, qv[2 * j], d);
                d = fmaf(f.y, qv[2 * j + 1], d);
            }
            d = warp_sum(d);
            s[u] = ok ? d : -INFINITY;
        }
        float mn = m;
#pragma unroll
        for (uint32_t u = 0; u < U4; u++) mn = fmaxf(mn, s[u]);
        const float alpha = expf(m - mn);
        l *= alpha;
#pragma unroll
        for (int d = 0; d < PL; d++) acc[d] *= alpha;
#pragma unroll
        for (uint32_t u = 0; u < U4; u++) {
            const float p = expf(s[u] - mn);
            l += p;
            const uint32_t w4[4] = {vv[u].x, vv[u].y, vv[u].z, vv[u].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(*(const __half2 *)&w4[j]);
                acc[2 * j] = fmaf(p, f.x, acc[2 * j]);
                acc[2 * j + 1] = fmaf(p, f.y, acc[2 * j + 1]);
            }
        }
        m = mn;
    }
    float *o = part + (((size_t)t * a.max_chunks + ch) * QH + qh) * (HD + 2);
#pragma unroll
    for (int d = 0; d < PL; d++) o[lane * PL + d] = acc[d];
    if (lane == 0) {
        o[HD] = m;
        o[HD + 1] = l;
    }
}

static cudaError_t launch_qsa_attn(const QwLaunch &L) {
    uint32_t QH, KVH, HD;
    QW_CHECK_ARG(qsa_dims(L, QH, KVH, HD));
    qsa_args a = L.bytes<qsa_args>(6);
    QW_CHECK_ARG(L.has_bytes(6, 24) && a.nb >= 1 && a.nb <= 64 && a.layer < a.nlayers && a.max_chunks >= 1 && a.max_chunks <= a.max_pages);
    for (int i = 0; i <= 5; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * QH * HD * 2 && L.avail(5) >= (size_t)a.nb * a.max_chunks * QH * (HD + 2) * 4 && L.tx == 256);
    qw_launch(qsa_attn_k, dim3(a.max_chunks, KVH, a.nb), 256, 0, L.stream, L.buf<__half>(0), L.buf<__half>(1), L.buf<int32_t>(2), L.buf<int32_t>(3),
                                                                   L.buf<int32_t>(4), L.buf<float>(5), a, QH, KVH);
    return cudaGetLastError();
}
QW_FAMILY(qsa_attn_simt, launch_qsa_attn, 256)

// ------------------------------------------------------------------------------------------------ attention core, tensor cores
// Same contract and partial format as qsa_attn_simt above, computed with warp MMAs on K / V tiles staged by 2-D
// tiled TMA copies (cp.async.bulk.tensor, 128-byte swizzle) -- this is the family the engine uses ("qsa_attn").
// Persistent warps: the (page chunk, kv head, slot) tasks of the launch are numbered slot-major and warp number w of the
// grid takes tasks w, w + W, w + 2W, ...  A warp owns a task completely: it walks the page's up to 256 tokens in steps
// of 16 with its own K and V tile and two mbarriers, keeps the online-softmax state of the 8 query heads in registers and
// writes the partial straight from them -- no block-wide synchronisation after the start, and the tiles of a warp's next
// task are requested while the current one finishes, so a warp always has a copy in flight.
//   scores   S^T[16 tokens][8 heads] = K[16][256] . Q^T            16 MMAs m16n8k16, A = K rows via ldmatrix
//   softmax  online, per head, over the token rows (lanes that share t = lane % 4 hold the same two heads)
//   output   O^T[256 dims][8 heads] += V^T[256][16 tokens] . P^T   16 MMAs, A = V via ldmatrix.trans,
//            B = the probabilities moved from accumulator layout to operand layout with four shuffles
// The 8 query heads of the kv head fill the MMA's N dimension exactly: nothing is padded.  What a task computes depends
// only on its slot's own length, never on which warp runs it or on the other slots of the batch.
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// STG = 1: one tile of K and one of V per warp and three blocks per SM -- many warps hide one another's copies.  STG = 3, for launches with
// no more tasks than one block per SM has warps: nobody else hides a warp's copies then, and with one tile in flight each of a page's 16
// steps waited a whole memory latency (1.3 us); three tiles of both in a ring.  Measured on a B200, step time with STG = 1 over step time
// with STG = 3, 12 layers: 1 slot of 6000 to 48000 tokens 1.04 to 1.03, 2 slots of 6000 to 36000 1.035 to 1.02, 3 of 3000 to 24000 1.03 to 1.02, 5 of 3000
// to 12000 and 8 of 1000 to 9000 1.00 to 1.01; a prompt's group of 64 rows in its first 1024 tokens (prep, core and merge alone) 1.20 to 1.29, of
// 8 rows in its first 4096 1.07 to 1.36.
constexpr int AT_TILE_BYTES = 16384;  // K tile 8 KB + V tile 8 KB (4 swizzled boxes of 16 rows x 128 B each)
constexpr int AT_TAB_BYTES = 896;     // per block: first task of every slot [65], tokens [64], slot id [64]
constexpr int AT_ZERO_BYTES = 3 * 2048 + 128;  // a row of zeros for each of a V tile's boxes, as far apart as the boxes
constexpr int AT_FEW_STG = 3;
constexpr int at_smem(int stg) { return 4 * stg * AT_TILE_BYTES + 128 + AT_TAB_BYTES + AT_ZERO_BYTES + 1024; }
constexpr int at_blocks_per_sm(int stg) { return stg == 1 ? 3 : 1; }  // what the shared memory and the registers of the kernel allow

template <int STG>
__global__ void __launch_bounds__(128) qsa_attn_mma_k(const __grid_constant__ CUtensorMap tm, const __half *q, const int32_t *pt, const int32_t *posv,
                                                      const int32_t *sids, float *part, qsa_args a, uint32_t QH, uint32_t KVH, unsigned *status) {
    constexpr uint32_t HD = 256;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    uint8_t *smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);  // swizzled boxes need 1024-byte alignment
    uint8_t *Kb = smem + warp * STG * AT_TILE_BYTES, *Vb = Kb + 8192;
    constexpr int NBAR = STG == 1 ? 2 : STG;  // STG = 1: K and V on their own; else one per tile pair
    uint64_t *bars = (uint64_t *)(smem + 4 * STG * AT_TILE_BYTES) + warp * NBAR;
    uint32_t *first = (uint32_t *)(smem + 4 * STG * AT_TILE_BYTES + 128), *ntokv = first + 65, *sidv = ntokv + 64;
    const uint32_t zeros = smem_u32(first) + AT_TAB_BYTES;
    first[(AT_TAB_BYTES + warp * 2048) / 4 + lane] = 0;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NBAR; k++) mbar_init(&bars[k], 1);
        mbar_init_fence();
    }
    pdl_sync();
    // pages of every slot and their running sum: slot s owns page numbers first[s] .. first[s + 1] - 1 of the launch
    if (warp == 0) {
        uint32_t c[2], nt[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t sl = lane + 32 * h;
            nt[h] = sl < a.nb ? (uint32_t)posv[sl] + 1 : 0;
            c[h] = min((nt[h] + QSA_PAGE - 1) / QSA_PAGE, a.max_chunks);
            ntokv[sl] = nt[h];
            sidv[sl] = sl < a.nb ? (uint32_t)sids[sl] : 0;
        }
        uint32_t s0 = c[0], s1 = c[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u0 = __shfl_up_sync(0xffffffffu, s0, o), u1 = __shfl_up_sync(0xffffffffu, s1, o);
            if (lane >= (uint32_t)o) {
                s0 += u0;
                s1 += u1;
            }
        }
        const uint32_t tot0 = __shfl_sync(0xffffffffu, s0, 31);
        first[lane] = s0 - c[0];
        first[32 + lane] = tot0 + s1 - c[1];
        if (lane == 31) first[64] = tot0 + s1;
    }
    __syncthreads();
    const uint32_t tasks = first[64] * KVH, W = gridDim.x * 4;
    struct Task {
        uint32_t ts, kvh, ch, n;
        int rowK;
    };
    auto task_of = [&](uint32_t i) {  // i < tasks
        Task k;
        const uint32_t pi = i / KVH;
        k.kvh = i - pi * KVH;
        uint32_t lo = 0, hi = a.nb;  // largest slot with first[slot] <= pi (every slot of the step has at least one page)
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (first[mid] <= pi) lo = mid;
            else hi = mid;
        }
        k.ts = lo;
        k.ch = pi - first[lo];
        k.n = min((uint32_t)QSA_PAGE, ntokv[lo] - k.ch * QSA_PAGE);
        const uint32_t page = (uint32_t)pt[(size_t)sidv[lo] * a.max_pages + k.ch];
        k.rowK = (int)(((page * a.nlayers + a.layer) * 2) * KVH * QSA_PAGE + k.kvh * QSA_PAGE);
        return k;
    };
    auto load = [&](uint8_t *dst, uint64_t *bar, int row) {
        if (lane == 0) {
            fence_proxy_async();  // the warp's reads of this buffer (ordered by __syncwarp) before the async-proxy writes
            mbar_expect_tx(bar, 8192);
#pragma unroll
            for (int db = 0; db < 4; db++) tma_load_2d(smem_u32(dst) + db * 2048, &tm, db * 64, row, bar);
        }
    };
    // ldmatrix lane roles: matrix mi = lane / 8, row r8 = lane % 8 (the swizzle key of that row)
    const uint32_t mi = lane >> 3, r8 = lane & 7;
    const uint32_t vrow = (mi >> 1) * 8 + r8;  // token of the V tile whose row this lane addresses
    const uint32_t kbase = smem_u32(Kb) + ((mi & 1) * 8 + r8) * 128, vbase = smem_u32(Vb) + vrow * 128;
    const int vrows = (int)(KVH * QSA_PAGE);  // rows from a page's K tile to its V tile
    uint32_t kph = 0, vph = 0;  // copies waited for so far on the K / V barrier (their parity selects the phase)
    bool ok = true;
    uint32_t i = STG == 1 ? blockIdx.x * 4 + warp : warp * gridDim.x + blockIdx.x;  // (few tasks go to different SMs first)
    Task cur{};
    // STG > 1: the ring is fed tile by tile over the warp's tasks, STG tiles ahead of the one in work (tile number n of the warp)
    uint32_t n = 0, fi = i, fs = 0;
    Task ft{};
    auto feed = [&](uint32_t at) {
        if (fi >= tasks) return;
        const uint32_t st = at % STG;
        if (lane == 0) {
            fence_proxy_async();  // the warp's reads of the stage (ordered by __syncwarp) before the async-proxy writes
            mbar_expect_tx(&bars[st], AT_TILE_BYTES);
#pragma unroll
            for (int db = 0; db < 4; db++) {
                tma_load_2d(smem_u32(Kb) + st * AT_TILE_BYTES + db * 2048, &tm, db * 64, ft.rowK + (int)fs * 16, &bars[st]);
                tma_load_2d(smem_u32(Vb) + st * AT_TILE_BYTES + db * 2048, &tm, db * 64, ft.rowK + vrows + (int)fs * 16, &bars[st]);
            }
        }
        if (++fs == (ft.n + 15) / 16) {
            fs = 0;
            fi += W;
            if (fi < tasks) ft = task_of(fi);
        }
    };
    if (i < tasks) {
        cur = task_of(i);
        if (STG == 1) {
            load(Kb, &bars[0], cur.rowK);
            load(Vb, &bars[1], cur.rowK + vrows);
        } else {
            ft = cur;
            for (uint32_t k = 0; k < STG; k++) feed(k);
        }
    }
    while (i < tasks && ok) {
        const uint32_t steps = (cur.n + 15) / 16;
        const bool more = i + W < tasks;
        Task nxt{};
        if (more) nxt = task_of(i + W);  // looked up now: its first tiles are requested as soon as this task's last ones are consumed
        // Q as B fragments (k = dim, n = head g), pre-scaled by HD^-1/2 = 1/16 (exact in fp16)
        uint32_t qf[16][2];
        {
            const __half *qp = q + ((size_t)cur.ts * QH + cur.kvh * 8 + g) * HD + 2 * t;
            const __half2 sc = __floats2half2_rn(0.0625f, 0.0625f);
#pragma unroll
            for (int ks = 0; ks < 16; ks++) {
                const __half2 v0 = __hmul2(*(const __half2 *)(qp + 16 * ks), sc), v1 = __hmul2(*(const __half2 *)(qp + 16 * ks + 8), sc);
                qf[ks][0] = *(const uint32_t *)&v0;
                qf[ks][1] = *(const uint32_t *)&v1;
            }
        }
        float o[16][4];
#pragma unroll
        for (int dt = 0; dt < 16; dt++) o[dt][0] = o[dt][1] = o[dt][2] = o[dt][3] = 0.f;
        float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
        for (uint32_t step = 0; step < steps; step++) {
            const uint32_t so = STG == 1 ? 0 : n % STG * AT_TILE_BYTES;
            if (!(STG == 1 ? mbar_wait(&bars[0], kph & 1) : mbar_wait(&bars[n % STG], n / STG & 1))) { ok = false; break; }
            kph++;
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < 16; ks++) {
                uint32_t af[4];
                ldsm_x4(af, kbase + so + (ks >> 2) * 2048 + ((((ks & 3) * 2 + (mi >> 1)) ^ r8) << 4));
                mma_f16(s, af, qf[ks][0], qf[ks][1], s);
            }
            if (STG == 1) {
                __syncwarp();
                if (step + 1 < steps) load(Kb, &bars[0], cur.rowK + (int)(step + 1) * 16);
                else if (more) load(Kb, &bars[0], nxt.rowK);
            }
            const uint32_t ta = step * 16 + g;
            if (ta >= cur.n) s[0] = s[1] = -INFINITY;
            if (ta + 8 >= cur.n) s[2] = s[3] = -INFINITY;
            float x0 = fmaxf(s[0], s[2]), x1 = fmaxf(s[1], s[3]);
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) {
                x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, off));
                x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, off));
            }
            const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
            const float a0 = expf(m0 - n0), a1 = expf(m1 - n1);
            const float p0 = expf(s[0] - n0), p1 = expf(s[1] - n1), p2 = expf(s[2] - n0), p3 = expf(s[3] - n1);
            l0 = l0 * a0 + (p0 + p2);
            l1 = l1 * a1 + (p1 + p3);
            m0 = n0;
            m1 = n1;
#pragma unroll
            for (int dt = 0; dt < 16; dt++) {
                o[dt][0] *= a0;
                o[dt][1] *= a1;
                o[dt][2] *= a0;
                o[dt][3] *= a1;
            }
            // probabilities: accumulator layout (token g / g+8, heads 2t, 2t+1) -> B operand layout (tokens 2t, 2t+1 / +8,
            // head g).  Each probability travels as an fp16 high part plus an fp16 remainder (two MMAs per dim tile), so the
            // weighted sum keeps ~22 bits of p instead of 11.
            const __half2 h01 = __floats2half2_rn(p0, p1), h23 = __floats2half2_rn(p2, p3);
            const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
            const __half2 r01 = __floats2half2_rn(p0 - f01.x, p1 - f01.y), r23 = __floats2half2_rn(p2 - f23.x, p3 - f23.y);
            const int srcA = (2 * t) * 4 + (g >> 1), srcB = srcA + 4;
            const uint32_t sel = (g & 1) ? 0x7632u : 0x5410u;
            auto to_b = [&](const __half2 &h) {
                const uint32_t u = *(const uint32_t *)&h;
                return __byte_perm(__shfl_sync(0xffffffffu, u, srcA), __shfl_sync(0xffffffffu, u, srcB), sel);
            };
            const uint32_t b0 = to_b(h01), b1 = to_b(h23), c0 = to_b(r01), c1 = to_b(r23);
            if (STG == 1 && !mbar_wait(&bars[1], vph & 1)) { ok = false; break; }
            vph++;
            // Rows of the tile past the slot's length: their probabilities are 0, but the page may hold anything there -- a later token of the same
            // prompt, or what an earlier conversation left -- and 0 times an infinity or a NaN would reach every head.  Lanes that address such a row
            // read zeros instead: one select per step, prep, core and merge of one slot of 6000 tokens 26.0 -> 26.3 us.  (Zeroing the tile's rows in
            // place: 26.8; a branch in the step keeps V's loads behind the softmax.)
            const uint32_t va = step * 16 + vrow < cur.n ? vbase + so : zeros;
            // four dim tiles at a time: the two MMAs of a tile depend on one another, back to back the second would wait for the first
#pragma unroll
            for (int dq = 0; dq < 4; dq++) {
                uint32_t af[4][4];
#pragma unroll
                for (int j = 0; j < 4; j++) ldsm_x4_t(af[j], va + dq * 2048 + (((j * 2 + (mi & 1)) ^ r8) << 4));
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f16(o[4 * dq + j], af[j], b0, b1, o[4 * dq + j]);
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f16(o[4 * dq + j], af[j], c0, c1, o[4 * dq + j]);
            }
            __syncwarp();
            if (STG > 1) {
                feed(n + STG);
                n++;
            } else if (step + 1 < steps) load(Vb, &bars[1], cur.rowK + vrows + (int)(step + 1) * 16);
            else if (more) load(Vb, &bars[1], nxt.rowK + vrows);
        }
        if (!ok) break;
        // the page's totals (the lanes that share t hold the same two heads), then the partial straight from the registers
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, off);
            l1 += __shfl_xor_sync(0xffffffffu, l1, off);
        }
        float *po0 = part + (((size_t)cur.ts * a.max_chunks + cur.ch) * QH + cur.kvh * 8 + 2 * t) * (HD + 2), *po1 = po0 + (HD + 2);
#pragma unroll
        for (int dt = 0; dt < 16; dt++) {
            po0[16 * dt + g] = o[dt][0];
            po1[16 * dt + g] = o[dt][1];
            po0[16 * dt + g + 8] = o[dt][2];
            po1[16 * dt + g + 8] = o[dt][3];
        }
        if (g == 0) {
            po0[HD] = m0;
            po0[HD + 1] = l0;
            po1[HD] = m1;
            po1[HD + 1] = l1;
        }
        cur = nxt;
        i += W;
    }
    if (!ok && lane == 0) set_status(status, ST_MBAR_TIMEOUT | 4);
}

// ---- The rows of a prompt's piece: up to a thousand queries of ONE slot.  Going by 64 rows, qsa_attn loads every page once per row and kv head -- 256 KB each,
// 20 us per launch -- although neighbouring rows read the same tiles.  Here a block is 16 rows of one (page, kv head): its tiles come once for all of them
// through a ring of four, and a warp runs two rows, so a fragment of K feeds two products and, below the rows' ends, a fragment of V too.
// A row's operations are those of qsa_attn_mma_k in the same order.  With the cache writes and the merges of all rows in one launch each, prompts of 12 layers on
// a B200: 419 tokens 7.58 -> 7.31 ms, 1024 15.2 -> 14.6, 1700 26.1 -> 25.0, 3000 45.3 -> 43.6.
// binds and partials as qsa_attn, sids[0] for all rows; ROWS = the most rows.  grid ceil(nb / 16) * max_chunks * KVH x 256
constexpr int AP_STG = 4, AP_WARPS = 8, AP_ROWS = 16;
constexpr int AP_SMEM = 1024 + AP_STG * AT_TILE_BYTES + AT_ZERO_BYTES + 2 * AP_STG * 8;
__global__ void __launch_bounds__(AP_WARPS * 32, 1) qsa_attn_piece_k(const __grid_constant__ CUtensorMap tm, const __half *q, const int32_t *pt, const int32_t *posv,
                                                                     const int32_t *sids, float *part, qsa_args a, uint32_t QH, uint32_t KVH, unsigned *status) {
    constexpr uint32_t HD = 256;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    uint8_t *smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    uint8_t *zrow = smem + AP_STG * AT_TILE_BYTES;
    uint64_t *full = (uint64_t *)(zrow + AT_ZERO_BYTES), *empty = full + AP_STG;
    const uint32_t base = smem_u32(smem), zeros = smem_u32(zrow);
    if (warp < 4) ((uint32_t *)zrow)[warp * 512 + lane] = 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < AP_STG; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], AP_WARPS);
        }
        mbar_init_fence();
    }
    pdl_sync();
    const uint32_t rb = blockIdx.x / (a.max_chunks * KVH), rem = blockIdx.x % (a.max_chunks * KVH), ch = rem / KVH, kvh = rem % KVH;
    // tokens of the page that a row attends to; the block walks as far as its longest row
    auto tokens_of = [&](uint32_t r) {
        const int n = r < a.nb ? posv[r] + 1 - (int)(ch * QSA_PAGE) : 0;
        return (uint32_t)(n < 0 ? 0 : n > QSA_PAGE ? QSA_PAGE : n);
    };
    const uint32_t r0 = rb * AP_ROWS + warp * 2;
    const uint32_t most = __reduce_max_sync(0xffffffffu, tokens_of(lane < AP_ROWS ? rb * AP_ROWS + lane : a.nb)), steps = (most + 15) / 16;
    const uint32_t n[2] = {tokens_of(r0), tokens_of(r0 + 1)};
    __syncthreads();
    if (steps == 0) return;
    const uint32_t page = (uint32_t)pt[(size_t)sids[0] * a.max_pages + ch];
    const int rowK = (int)(((page * a.nlayers + a.layer) * 2) * KVH * QSA_PAGE + kvh * QSA_PAGE), rowV = rowK + (int)(KVH * QSA_PAGE);
    auto put = [&](uint32_t j) {  // tile pair j; by one thread
        const uint32_t st = j % AP_STG;
        if (j >= AP_STG && !mbar_wait(&empty[st], (j / AP_STG - 1) & 1)) return false;
        fence_proxy_async();  // the warps' reads of the stage before the async-proxy writes
        mbar_expect_tx(&full[st], AT_TILE_BYTES);
#pragma unroll
        for (int db = 0; db < 4; db++) {
            tma_load_2d(base + st * AT_TILE_BYTES + db * 2048, &tm, db * 64, rowK + (int)j * 16, &full[st]);
            tma_load_2d(base + st * AT_TILE_BYTES + 8192 + db * 2048, &tm, db * 64, rowV + (int)j * 16, &full[st]);
        }
        return true;
    };
    if (threadIdx.x == 0)
        for (uint32_t j = 0; j < AP_STG - 1 && j < steps; j++) put(j);
    // Q of both rows as B fragments (k = dim, n = head g), pre-scaled by HD^-1/2 = 1/16 (exact in fp16)
    uint32_t qf[2][16][2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const __half *qp = q + ((size_t)(r0 + i < a.nb ? r0 + i : a.nb - 1) * QH + kvh * 8 + g) * HD + 2 * t;
        const __half2 sc = __floats2half2_rn(0.0625f, 0.0625f);
#pragma unroll
        for (int ks = 0; ks < 16; ks++) {
            const __half2 v0 = __hmul2(*(const __half2 *)(qp + 16 * ks), sc), v1 = __hmul2(*(const __half2 *)(qp + 16 * ks + 8), sc);
            qf[i][ks][0] = *(const uint32_t *)&v0;
            qf[i][ks][1] = *(const uint32_t *)&v1;
        }
    }
    const uint32_t mi = lane >> 3, r8 = lane & 7, vrow = (mi >> 1) * 8 + r8;
    const uint32_t kbase = base + ((mi & 1) * 8 + r8) * 128, vbase = base + 8192 + vrow * 128;
    float o[2][16][4], m[2][2], l[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
#pragma unroll
        for (int dt = 0; dt < 16; dt++) o[i][dt][0] = o[i][dt][1] = o[i][dt][2] = o[i][dt][3] = 0.f;
        m[i][0] = m[i][1] = -INFINITY;
        l[i][0] = l[i][1] = 0.f;
    }
    bool ok = true;
#pragma unroll 1
    for (uint32_t step = 0; step < steps; step++) {
        if (warp == 0) {  // three steps ahead, into the stage that every warp has left by now or leaves soon
            if (lane == 0 && step + AP_STG - 1 < steps) ok = put(step + AP_STG - 1);
            ok = __shfl_sync(0xffffffffu, (int)ok, 0);
        }
        const uint32_t st = step % AP_STG, so = st * AT_TILE_BYTES;
        ok = ok && mbar_wait(&full[st], (step / AP_STG) & 1);
        if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            // no block ends with copies of its own in flight: those that may be are waited for, with a limit again
            if (threadIdx.x == 0)
                for (uint32_t j = step; j < steps && j < step + AP_STG; j++) mbar_wait(&full[j % AP_STG], (j / AP_STG) & 1);
            break;
        }
        const bool on0 = step * 16 < n[0], on1 = step * 16 < n[1];  // (the same in all lanes)
        if (on0 || on1) {
            float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int ks = 0; ks < 16; ks++) {
                uint32_t af[4];
                ldsm_x4(af, kbase + so + (ks >> 2) * 2048 + ((((ks & 3) * 2 + (mi >> 1)) ^ r8) << 4));
                mma_f16(s[0], af, qf[0][ks][0], qf[0][ks][1], s[0]);
                mma_f16(s[1], af, qf[1][ks][0], qf[1][ks][1], s[1]);
            }
            uint32_t pb[2][4];  // probabilities as B operands: high parts, remainders
            const uint32_t ta = step * 16 + g;
            auto softmax = [&](int i) {
                if (ta >= n[i]) s[i][0] = s[i][1] = -INFINITY;
                if (ta + 8 >= n[i]) s[i][2] = s[i][3] = -INFINITY;
                float x0 = fmaxf(s[i][0], s[i][2]), x1 = fmaxf(s[i][1], s[i][3]);
#pragma unroll
                for (int off = 4; off < 32; off <<= 1) {
                    x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, off));
                    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, off));
                }
                const float n0 = fmaxf(m[i][0], x0), n1 = fmaxf(m[i][1], x1);
                const float a0 = expf(m[i][0] - n0), a1 = expf(m[i][1] - n1);
                const float p0 = expf(s[i][0] - n0), p1 = expf(s[i][1] - n1), p2 = expf(s[i][2] - n0), p3 = expf(s[i][3] - n1);
                l[i][0] = l[i][0] * a0 + (p0 + p2);
                l[i][1] = l[i][1] * a1 + (p1 + p3);
                m[i][0] = n0;
                m[i][1] = n1;
#pragma unroll
                for (int dt = 0; dt < 16; dt++) {
                    o[i][dt][0] *= a0;
                    o[i][dt][1] *= a1;
                    o[i][dt][2] *= a0;
                    o[i][dt][3] *= a1;
                }
                const __half2 h01 = __floats2half2_rn(p0, p1), h23 = __floats2half2_rn(p2, p3);
                const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
                const __half2 e01 = __floats2half2_rn(p0 - f01.x, p1 - f01.y), e23 = __floats2half2_rn(p2 - f23.x, p3 - f23.y);
                const int srcA = (2 * t) * 4 + (g >> 1), srcB = srcA + 4;
                const uint32_t sel = (g & 1) ? 0x7632u : 0x5410u;
                auto to_b = [&](const __half2 &h) {
                    const uint32_t u = *(const uint32_t *)&h;
                    return __byte_perm(__shfl_sync(0xffffffffu, u, srcA), __shfl_sync(0xffffffffu, u, srcB), sel);
                };
                pb[i][0] = to_b(h01);
                pb[i][1] = to_b(h23);
                pb[i][2] = to_b(e01);
                pb[i][3] = to_b(e23);
            };
            auto value_of = [&](int i, int dq, const uint32_t (&af)[4][4]) {
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f16(o[i][4 * dq + j], af[j], pb[i][0], pb[i][1], o[i][4 * dq + j]);
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f16(o[i][4 * dq + j], af[j], pb[i][2], pb[i][3], o[i][4 * dq + j]);
            };
            auto v_frag = [&](uint32_t (&af)[4][4], uint32_t va, int dq) {
#pragma unroll
                for (int j = 0; j < 4; j++) ldsm_x4_t(af[j], va + dq * 2048 + (((j * 2 + (mi & 1)) ^ r8) << 4));
            };
            if (step * 16 + 16 <= n[0] && step * 16 + 16 <= n[1]) {  // both rows see the whole tile
                softmax(0);
                softmax(1);
#pragma unroll
                for (int dq = 0; dq < 4; dq++) {
                    uint32_t af[4][4];
                    v_frag(af, vbase + so, dq);
                    value_of(0, dq, af);
                    value_of(1, dq, af);
                }
            } else {  // the tile in which a row ends: rows of V past it are read as zeros, whatever the page holds there
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    if (!(i ? on1 : on0)) continue;
                    softmax(i);
                    const uint32_t va = step * 16 + vrow < n[i] ? vbase + so : zeros;
#pragma unroll
                    for (int dq = 0; dq < 4; dq++) {
                        uint32_t af[4][4];
                        v_frag(af, va, dq);
                        value_of(i, dq, af);
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[st]);
    }
    if (!ok) {
        if (lane == 0) set_status(status, ST_MBAR_TIMEOUT | 17);
        return;
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (n[i] == 0) continue;
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            l[i][0] += __shfl_xor_sync(0xffffffffu, l[i][0], off);
            l[i][1] += __shfl_xor_sync(0xffffffffu, l[i][1], off);
        }
        float *po0 = part + (((size_t)(r0 + i) * a.max_chunks + ch) * QH + kvh * 8 + 2 * t) * (HD + 2), *po1 = po0 + (HD + 2);
#pragma unroll
        for (int dt = 0; dt < 16; dt++) {
            po0[16 * dt + g] = o[i][dt][0];
            po1[16 * dt + g] = o[i][dt][1];
            po0[16 * dt + g + 8] = o[i][dt][2];
            po1[16 * dt + g + 8] = o[i][dt][3];
        }
        if (g == 0) {
            po0[HD] = m[i][0];
            po0[HD + 1] = l[i][0];
            po1[HD] = m[i][1];
            po1[HD + 1] = l[i][1];
        }
    }
}

// The pool seen as [rows of one token of one kv head][256 halves]
static bool attn_encode_map(CUtensorMap *tm, const void *pool, size_t bytes) {
    return tmap_2d(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, pool, 256, bytes / 512, 512, 64, 16, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
}

// One tensor map per KV pool
static const CUtensorMap *attn_tensor_map(void *pool, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<void *, size_t>, CUtensorMap> cache;
    std::lock_guard<std::mutex> lk(mu);
    auto key = std::make_pair(pool, bytes);
    auto it = cache.find(key);
    if (it != cache.end()) return &it->second;
    CUtensorMap tm;
    if (!attn_encode_map(&tm, pool, bytes)) return nullptr;
    return &(cache[key] = tm);
}

// Persistent: as many blocks as fit on the device at once, or fewer when the step cannot have that many tasks.  most = the most tasks the
// launch can have (slots x chunks x kv heads); with up to one per warp of a block on every SM the deep ring is the faster form.
struct AttnLaunch {
    decltype(&qsa_attn_mma_k<1>) k;
    uint32_t grid;
    int smem;
};
static AttnLaunch attn_launch(uint32_t most, uint32_t sms) {
    if (most <= 4 * sms) return {qsa_attn_mma_k<AT_FEW_STG>, most < sms ? most : sms, at_smem(AT_FEW_STG)};
    const uint32_t blocks = (most + 3) / 4, cap = sms * at_blocks_per_sm(1);
    return {qsa_attn_mma_k<1>, blocks < cap ? blocks : cap, at_smem(1)};
}

static cudaError_t launch_qsa_attn_piece(const QwLaunch &L) {
    uint32_t QH, KVH, HD;
    QW_CHECK_ARG(qsa_dims(L, QH, KVH, HD));
    qsa_args a = L.bytes<qsa_args>(6);
    QW_CHECK_ARG(L.has_bytes(6, 24) && a.nb >= 1 && a.nb <= (uint32_t)L.def("ROWS", 64) && a.layer < a.nlayers && a.max_chunks >= 1 && a.max_chunks <= a.max_pages);
    for (int i = 0; i <= 5; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * QH * HD * 2 && L.avail(3) >= (size_t)a.nb * 4 && L.avail(4) >= 4 &&
                 L.avail(5) >= (size_t)a.nb * a.max_chunks * QH * (HD + 2) * 4);
    QW_CHECK_ARG(((uintptr_t)L.buf<void>(1) & 15) == 0 && L.avail(1) >= 512 && L.avail(1) / 512 < 0x7fffffffull);
    const CUtensorMap *tm = attn_tensor_map(L.buf<void>(1), L.avail(1) / 512 * 512);
    QW_CHECK_ARG(tm != nullptr);
    const cudaError_t e = cudaFuncSetAttribute(qsa_attn_piece_k, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMEM);
    if (e != cudaSuccess) return e;
    qw_launch(qsa_attn_piece_k, (a.nb + AP_ROWS - 1) / AP_ROWS * a.max_chunks * KVH, AP_WARPS * 32, AP_SMEM, L.stream, *tm, L.buf<__half>(0), L.buf<int32_t>(2), L.buf<int32_t>(3),
              L.buf<int32_t>(4), L.buf<float>(5), a, QH, KVH, L.status);
    return cudaGetLastError();
}
QW_FAMILY(qsa_attn_piece, launch_qsa_attn_piece, 256)

static cudaError_t launch_qsa_attn_mma(const QwLaunch &L) {
    uint32_t QH, KVH, HD;
    QW_CHECK_ARG(qsa_dims(L, QH, KVH, HD));
    qsa_args a = L.bytes<qsa_args>(6);
    QW_CHECK_ARG(L.has_bytes(6, 24) && a.nb >= 1 && a.nb <= 64 && a.layer < a.nlayers && a.max_chunks >= 1 && a.max_chunks <= a.max_pages);
    for (int i = 0; i <= 5; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * QH * HD * 2 && L.avail(5) >= (size_t)a.nb * a.max_chunks * QH * (HD + 2) * 4);
    QW_CHECK_ARG(((uintptr_t)L.buf<void>(1) & 15) == 0 && L.avail(1) >= 512 && L.avail(1) / 512 < 0x7fffffffull);
    const CUtensorMap *tm = attn_tensor_map(L.buf<void>(1), L.avail(1) / 512 * 512);
    QW_CHECK_ARG(tm != nullptr);
    const AttnLaunch at = attn_launch(a.nb * a.max_chunks * KVH, (uint32_t)L.sm_count);
    const cudaError_t e = cudaFuncSetAttribute(at.k, cudaFuncAttributeMaxDynamicSharedMemorySize, at.smem);
    if (e != cudaSuccess) return e;
    qw_launch(at.k, at.grid, 128, at.smem, L.stream, *tm, L.buf<__half>(0), L.buf<int32_t>(2), L.buf<int32_t>(3), L.buf<int32_t>(4), L.buf<float>(5), a, QH, KVH, L.status);
    return cudaGetLastError();
}
QW_FAMILY(qsa_attn, launch_qsa_attn_mma, 128)

// ------------------------------------------------------------------------------------------------ merge + output gate
// binds: 0 = part, 1 = qkv fp16 (gate = qkv[t][qh*2*HD + HD + d]), 2 = y fp16 [nb][QH*HD], 3 = pos, 4 = qsa_args.
// grid (QH, nb) x 512.  The chunk weights exp(m_c - M) are computed once per chunk (thread c); then the 16 warps take the
// chunks c = warp, warp + 16, ... (each in increasing order; a lane owns eight dims: four 8-byte loads per chunk -- a partial's 258
// floats keep rows 8-byte aligned, not 16 -- four chunks in flight per warp) and the 16 partial sums are added in warp order: o = sum_c w_c acc_c[d] / sum_c w_c l_c.  The order depends only on the slot's own chunk count.
#define QSA_MAXCH 1024
__global__ void __launch_bounds__(512) qsa_merge_k(const float *part, const __half *qkv, __half *y, const int32_t *posv, qsa_args a, uint32_t QH) {
    constexpr uint32_t HD = 256;
    __shared__ float wc[QSA_MAXCH], lc[QSA_MAXCH], tmp[16], ls[16];
    __shared__ float accs[16][HD];
    pdl_sync();
    const uint32_t qh = blockIdx.x, t = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the core wrote max_chunks partials per slot at most: a position beyond that (only a caller that passes its own device
    // positions can produce one) must not make the merge read another slot's partials or run off the buffer
    const uint32_t ntok = (uint32_t)posv[t] + 1, nch = min((ntok + QSA_PAGE - 1) / QSA_PAGE, min(a.max_chunks, (uint32_t)QSA_MAXCH));
    const float *base = part + ((size_t)t * a.max_chunks * QH + qh) * (HD + 2);
    const size_t cstride = (size_t)QH * (HD + 2);
    float mx = -INFINITY;
    for (uint32_t c = tid; c < nch; c += 512) {
        const float pm = base[c * cstride + HD], pl = base[c * cstride + HD + 1];
        wc[c] = pm;
        lc[c] = pl;
        if (pl > 0.f) mx = fmaxf(mx, pm);
    }
    mx = warp_max(mx);
    if (lane == 0) tmp[warp] = mx;
    __syncthreads();
    float M = tmp[0];
#pragma unroll
    for (int i = 1; i < 16; i++) M = fmaxf(M, tmp[i]);
    for (uint32_t c = tid; c < nch; c += 512) wc[c] = lc[c] > 0.f ? expf(wc[c] - M) : 0.f;
    __syncthreads();
    float l = 0.f;
    float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 4
    for (uint32_t c = warp; c < nch; c += 16) {
        const float w = wc[c];
        const float2 *pv = (const float2 *)(base + c * cstride) + 4 * lane;
        const float2 v0 = pv[0], v1 = pv[1], v2 = pv[2], v3 = pv[3];
        l = fmaf(lc[c], w, l);
        acc[0].x = fmaf(v0.x, w, acc[0].x); acc[0].y = fmaf(v0.y, w, acc[0].y);
        acc[1].x = fmaf(v1.x, w, acc[1].x); acc[1].y = fmaf(v1.y, w, acc[1].y);
        acc[2].x = fmaf(v2.x, w, acc[2].x); acc[2].y = fmaf(v2.y, w, acc[2].y);
        acc[3].x = fmaf(v3.x, w, acc[3].x); acc[3].y = fmaf(v3.y, w, acc[3].y);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) *(float2 *)&accs[warp][8 * lane + 2 * i] = acc[i];
    if (lane == 0) ls[warp] = l;
    __syncthreads();
    if (tid < HD) {
        const uint32_t d = tid;
        float at = accs[0][d], lt = ls[0];
#pragma unroll
        for (int g2 = 1; g2 < 16; g2++) {
            at += accs[g2][d];
            lt += ls[g2];
        }
        const float g = __half2float(qkv[(size_t)t * a.qkv_stride + qh * 2 * HD + HD + d]);
        const float o = __half2float(__float2half_rn(at / lt));
        y[((size_t)t * QH + qh) * HD + d] = __float2half_rn(o * (1.0f / (1.0f + expf(-g))));
    }
}

// Many rows of few chunks (a prompt's piece, at most 16 pages): a warp per head and row, eight dims per lane.  The 16 groups of qsa_merge_k are then the chunks
// themselves, added in order; absent ones add zero, as there.  grid ceil(QH nb / 8) x 256
__global__ void __launch_bounds__(256) qsa_merge_rows_k(const float *part, const __half *qkv, __half *y, const int32_t *posv, qsa_args a, uint32_t QH) {
    constexpr uint32_t HD = 256;
    pdl_sync();
    const uint32_t n = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, t = n / QH, qh = n % QH;
    if (t >= a.nb) return;
    const uint32_t ntok = (uint32_t)posv[t] + 1, nch = min((ntok + QSA_PAGE - 1) / QSA_PAGE, a.max_chunks);
    const float *base = part + ((size_t)t * a.max_chunks * QH + qh) * (HD + 2);
    const size_t cstride = (size_t)QH * (HD + 2);
    const float pm = lane < nch ? base[lane * cstride + HD] : 0.f, pl = lane < nch ? base[lane * cstride + HD + 1] : 0.f;
    const float M = warp_max(pl > 0.f ? pm : -INFINITY);
    const float w = pl > 0.f ? expf(pm - M) : 0.f;
    float lt = 0.f, at[8];
#pragma unroll
    for (uint32_t c = 0; c < 16; c++) {
        const float wc = __shfl_sync(0xffffffffu, w, c), lc = __shfl_sync(0xffffffffu, pl, c);
        float x[8], lx = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = 0.f;
        if (c < nch) {  // (the same in all lanes)
            const float2 *pv = (const float2 *)(base + c * cstride) + 4 * lane;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 v = pv[i];
                x[2 * i] = fmaf(v.x, wc, 0.f);
                x[2 * i + 1] = fmaf(v.y, wc, 0.f);
            }
            lx = fmaf(lc, wc, 0.f);
        }
        lt = c ? lt + lx : lx;
#pragma unroll
        for (int i = 0; i < 8; i++) at[i] = c ? at[i] + x[i] : x[i];
    }
    const __half *gp = qkv + (size_t)t * a.qkv_stride + qh * 2 * HD + HD + 8 * lane;
    __half *yp = y + ((size_t)t * QH + qh) * HD + 8 * lane;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float g = __half2float(gp[i]);
        const float o = __half2float(__float2half_rn(at[i] / lt));
        yp[i] = __float2half_rn(o * (1.0f / (1.0f + expf(-g))));
    }
}

static cudaError_t launch_qsa_merge(const QwLaunch &L) {
    uint32_t QH, KVH, HD;
    QW_CHECK_ARG(qsa_dims(L, QH, KVH, HD));
    qsa_args a = L.bytes<qsa_args>(4);
    QW_CHECK_ARG(L.has_bytes(4, 24) && a.nb >= 1 && a.nb <= (uint32_t)L.def("ROWS", 64) && a.max_chunks >= 1 && a.max_chunks <= QSA_MAXCH);
    for (int i = 0; i <= 3; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * a.max_chunks * QH * (HD + 2) * 4 && L.avail(2) >= (size_t)a.nb * QH * HD * 2 &&
                 L.avail(1) >= ((size_t)(a.nb - 1) * a.qkv_stride + QH * 2 * HD) * 2);
    if (a.nb > 64 && a.max_chunks <= 16) {
        qw_launch(qsa_merge_rows_k, (QH * a.nb + 7) / 8, 256, 0, L.stream, L.buf<float>(0), L.buf<__half>(1), L.buf<__half>(2), L.buf<int32_t>(3), a, QH);
        return cudaGetLastError();
    }
    qw_launch(qsa_merge_k, dim3(QH, a.nb), 512, 0, L.stream, L.buf<float>(0), L.buf<__half>(1), L.buf<__half>(2), L.buf<int32_t>(3), a, QH);
    return cudaGetLastError();
}
QW_FAMILY(qsa_merge, launch_qsa_merge, 256)

// ------------------------------------------------------------------------------------------------ no-allocation entry point
// qw_attn_decode_static: the attention core + merge for callers that must not allocate device memory at all --
// for example code running inside someone else's memory plan (a serving process whose whole HBM budget was handed
// out at start-up, or a host that calls in while a stream capture is open elsewhere and therefore cannot call
// cudaMalloc).  The split-K partials, which the batch path keeps in a caller-provided buffer, live here in a
// file-scope device array; every GPU that loads this library holds that array (8.45 MB) until the process exits.
//
//   limit     nb * max_chunks <= QW_ATTN_STATIC_MAX_CHUNK_SLOTS (512 page-chunks in flight, e.g. 16 slots of up to
//             8192 tokens, or 2 slots of 65536); QH = 16, KVH = 2, HD = 256 only.  Larger requests are rejected.
//   set-up    the first call on a device resolves the array's device address (cudaGetSymbolAddress, with that
//             device current) and remembers it; make that first call outside any stream capture.
//   contract  pos[t] + 1 <= max_chunks * 256 for every row: the core covers max_chunks pages per slot and the merge never
//             looks past them (a longer position is cut to the first max_chunks pages, not read out of bounds).
//   contents  nothing has to start at zero: the core writes every partial (accumulator, max, sum) that the merge
//             of the same call reads, so what an earlier call left behind is never looked at.
//   sharing   all calls on a device use the same array: two calls whose kernels overlap on the GPU (different
//             streams, or different host threads) race and corrupt each other's result.  Serialise them.
// No cudaMalloc / cudaFree / host allocation happens on this path: the tensor map is encoded on the stack, the
// per-device address table is a static array.
#define QW_ATTN_STATIC_MAX_CHUNK_SLOTS 512
static __device__ __align__(256) float g_attn_static_part[(size_t)QW_ATTN_STATIC_MAX_CHUNK_SLOTS * 16 * (256 + 2)];
static float *g_attn_static_ptr[64];  // per device: address of the array above (host code may not use the symbol itself)

extern "C" int qw_attn_decode_static(const void *q, const void *kv_pool, size_t kv_pool_bytes, const int32_t *page_table, const int32_t *pos,
                                     const int32_t *slot_ids, const void *qkv, void *y, uint32_t nb, uint32_t layer, uint32_t nlayers,
                                     uint32_t qkv_stride, uint32_t max_pages, uint32_t max_chunks, void *stream, char *err, size_t errlen) {
    auto fail = [&](int code, const char *msg) {
        if (err && errlen) snprintf(err, errlen, "qw_attn_decode_static: %s", msg);
        return code;
    };
    constexpr uint32_t QH = 16, KVH = 2, HD = 256;
    if (!q || !kv_pool || !page_table || !pos || !slot_ids || !qkv || !y) return fail(-1, "null pointer argument");
    if (nb < 1 || nb > 64 || max_chunks < 1 || max_chunks > max_pages || layer >= nlayers) return fail(-1, "bad nb / max_chunks / layer");
    if ((uint64_t)nb * max_chunks > QW_ATTN_STATIC_MAX_CHUNK_SLOTS)
        return fail(-2, "nb * max_chunks exceeds the static scratch (512 page-chunks); use the batch path with a caller-provided buffer");
    if (qkv_stride < QH * 2 * HD + 2 * KVH * HD || ((uintptr_t)kv_pool & 15) || kv_pool_bytes < 512 || kv_pool_bytes / 512 >= 0x7fffffffull)
        return fail(-1, "bad qkv stride or KV pool");
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(-3, "no current CUDA device");
    if (!g_attn_static_ptr[dev]) {  // once per device, with that device current
        float *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress((void **)&p, g_attn_static_part);
        if (e != cudaSuccess || !p) return fail(-3, cudaGetErrorString(e));
        g_attn_static_ptr[dev] = p;
    }
    float *part = g_attn_static_ptr[dev];
    CUtensorMap tm;  // encoded on the stack: no allocation
    if (!attn_encode_map(&tm, kv_pool, kv_pool_bytes / 512 * 512)) return fail(-3, "tensor map encoding failed");
    qsa_args a = {nb, layer, nlayers, qkv_stride, max_pages, max_chunks, 0, 0};
    cudaStream_t st = (cudaStream_t)stream;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return fail(-3, "cannot read the SM count");
    const AttnLaunch at = attn_launch(nb * max_chunks * KVH, (uint32_t)sms);
    cudaError_t e = cudaFuncSetAttribute(at.k, cudaFuncAttributeMaxDynamicSharedMemorySize, at.smem);
    if (e != cudaSuccess) return fail(-3, cudaGetErrorString(e));
    at.k<<<at.grid, 128, at.smem, st>>>(tm, (const __half *)q, page_table, pos, slot_ids, part, a, QH, KVH, nullptr);
    qsa_merge_k<<<dim3(QH, nb), 512, 0, st>>>(part, (const __half *)qkv, (__half *)y, pos, a, QH);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(-3, cudaGetErrorString(e));
    if (err && errlen) err[0] = 0;
    return 0;
}
