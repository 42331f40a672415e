// Small kernels around the four big ones: embedding gather, residual add + RMSNorm, greedy arg-max, slot
// bookkeeping, buffer fill.
//   kb_embed     h[t] = float(emb[tok[t]])                       -- role of gg_embed / kb_embed (src/engine.c:8887-8898)
//   add_rmsnorm  h += delta (optional); x = fp16(h * rsqrt(mean h^2 + 1e-6) * w): the plain residual + RMSNorm
//                that stands in for the reference's hyper-connection mix (eps as every reference norm,
//                kernels/engine.metal:11)
//   k_argmax     per token arg-max over the vocabulary, equal values -> smallest index
//                -- role of k_argmax1/2 (kernels/engine.metal:605-648) and argmax_cpu (src/engine.c:6144-6148)
//   par_advance  after a step: pos[t] += 1 and (optionally) tok[t] = the sampled id, so consecutive greedy steps
//                need no host round trip
//   qw_fill      zero / counter-based synthetic fill of a buffer (weights of the synthetic model)
#include "common.cuh"
#include "moe_sel.h"
#include "qw_kern.h"
#include <cooperative_groups.h>

using namespace qw;

// binds: 0 = emb fp16 [V][D], 1 = tok int32 [nb], 2 = h fp32 [nb][D], 3 = {nb, D, V}.  grid (ceil(D/256), nb) x 256
__global__ void kb_embed_k(const __half *emb, const int32_t *tok, float *h, uint32_t D, uint32_t V) {
    pdl_sync();
    const uint32_t d = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
    if (d >= D) return;
    uint32_t id = (uint32_t)tok[t];
    if (id >= V) id = 0;
    h[(size_t)t * D + d] = __half2float(emb[(size_t)id * D + d]);
}
static cudaError_t launch_kb_embed(const QwLaunch &L) {
    struct { uint32_t nb, D, V; } a = L.bytes<decltype(a)>(3);
    QW_CHECK_ARG(L.buf<void>(0) && L.buf<void>(1) && L.buf<void>(2) && L.has_bytes(3, 12) && a.nb >= 1 && a.nb <= (uint32_t)L.def("ROWS", 64));
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.V * a.D * 2 && L.avail(1) >= a.nb * 4 && L.avail(2) >= (size_t)a.nb * a.D * 4);
    qw_launch(kb_embed_k, dim3((a.D + 255) / 256, a.nb), 256, 0, L.stream, L.buf<__half>(0), L.buf<int32_t>(1), L.buf<float>(2), a.D, a.V);
    return cudaGetLastError();
}
QW_FAMILY(kb_embed, launch_kb_embed, 256)

// binds: 0 = h fp32 [nb][D], 1 = delta fp16 [nb][D] (only with ADD defined 1: h is then updated in place),
// 2 = w fp32 [D], 3 = x out fp16 [nb][D], 4 = {nb, D}.  With CMB defined 1 the delta is not read from memory but is
// the MoE combine of moe_cmb (rank-ordered weighted sum of Pg plus the shared expert, rounded to fp16) computed on
// the fly: 5 = moe_sel, 6 = Pg fp32 [nb][TOPK+1][D], define TOPK.  ROWS = the most rows (default 64); WIDE defined 1: bind 5 is a
// moe_sel_wide.  grid nb x 256
template <int MODE>  // 0: norm only, 1: h += delta, 2: h += fp16(combine)
__global__ void __launch_bounds__(1024) add_rmsnorm_k(float *h, const __half *delta, const float *w, __half *x, uint32_t D, const moe_sel *ms,
                                                     const float *Pg, uint32_t topk, const unsigned *flags, const unsigned *seq, uint32_t nranks,
                                                     unsigned *status) {
    __shared__ float tmp[32];
    const uint32_t t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    pdl_launch();
    float wv[4];  // the norm weights are static: read before the wait for the previous kernel
#pragma unroll
    for (int it = 0; it < 4; it++) wv[it] = tid + it * nth < D ? w[tid + it * nth] : 0.f;
    pdl_wait();
    // rows of Pg (MODE 2) or of delta (MODE 1) may have been stored by other ranks: wait until every rank has published
    if (nranks > 1) ep_wait(flags, seq, nranks, status);
    float *hr = h + (size_t)t * D;
    float wk[MOE_MAXK];
    if (MODE == 2) {
        const float *wr = &ms->w[0][0] + t * (MOE_MAXK + 1);  // (moe_sel and moe_sel_wide keep w in the same place)
#pragma unroll
        for (uint32_t s = 0; s < MOE_MAXK; s++) wk[s] = s <= topk ? wr[s] : 0.f;
    }
    // a thread's values stay in registers between the two passes (D <= 4 * blockDim; beyond that they are read back)
    float vv[4] = {0.f, 0.f, 0.f, 0.f};
    float ss = 0.f;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const uint32_t d = tid + it * nth;
        if (d < D) {
            float v = hr[d];
            if (MODE == 1) {
                v += __half2float(delta[(size_t)t * D + d]);
                hr[d] = v;
            } else if (MODE == 2) {
                float pv[MOE_MAXK];  // all loads first (independent), then the rank-ordered chain
#pragma unroll
                for (uint32_t s = 0; s < MOE_MAXK; s++) pv[s] = s <= topk ? Pg[((size_t)t * (topk + 1) + s) * D + d] : 0.f;
                float o = 0.f;
#pragma unroll
                for (uint32_t s = 0; s < MOE_MAXK; s++)
                    if (s <= topk) o = fmaf(wk[s], pv[s], o);
                v += __half2float(__float2half_rn(o));
                hr[d] = v;
            }
            vv[it] = v;
            ss = fmaf(v, v, ss);
        }
    }
    for (uint32_t d = tid + 4 * nth; d < D; d += nth) {  // rows wider than the register copy
        float v = hr[d];
        if (MODE == 1) {
            v += __half2float(delta[(size_t)t * D + d]);
            hr[d] = v;
        } else if (MODE == 2) {
            float o = 0.f;
            for (uint32_t s = 0; s <= topk; s++) o = fmaf(wk[s], Pg[((size_t)t * (topk + 1) + s) * D + d], o);
            v += __half2float(__float2half_rn(o));
            hr[d] = v;
        }
        ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) tmp[warp] = ss;
    __syncthreads();
    const float tot = warp_sum(lane < nth / 32 ? tmp[lane] : 0.f);  // every warp sums the same 32 values in the same order
    const float r = rsqrtf(tot / D + 1e-6f);
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const uint32_t d = tid + it * nth;
        if (d < D) x[(size_t)t * D + d] = __float2half_rn(vv[it] * r * wv[it]);
    }
    for (uint32_t d = tid + 4 * nth; d < D; d += nth) x[(size_t)t * D + d] = __float2half_rn(hr[d] * r * w[d]);
}
// The MoE-combine form for D = 2048 (the step's hot case: it sits between the expert FFN and the next projection, and
// nothing else can run beside it).  A token is served by a cluster of 8 blocks of 256 threads, one column per thread: the
// twelve loads of a column are independent, the blocks are small enough to be resident next to the FFN's blocks while they
// wait for it, and the sum of squares of the row meets through the cluster's shared memory (every block pushes its partial sum to
// all eight; they are added in block order by every block, so the result does not depend on timing).  grid (8 nb) x 256, cluster 8.
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(256) cmb_rmsnorm_cl_k(float *h, const float *w, __half *x, const moe_sel *ms, const float *Pg,
                                                                                    uint32_t topk, const unsigned *flags, const unsigned *seq,
                                                                                    uint32_t nranks, unsigned *rowcnt, unsigned *status) {
    constexpr uint32_t D = 2048;
    namespace cg = cooperative_groups;
    __shared__ float tmp[8];
    __shared__ float parts[8];  // the eight blocks' partial sums of squares, each written here by its owner
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t t = blockIdx.x >> 3, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = (blockIdx.x & 7) * 256 + tid;
    pdl_launch();
    // first cluster barrier, split: arrive now, wait just before the partial sums are pushed (by then every block of the cluster
    // has long arrived, i.e. has started and owns its shared memory)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const float wd = w[d];  // the norm weights are static
    if (rowcnt) {
        // One GPU, the one-launch expert FFN before us: do not wait for its whole launch, only for this token's topk + 1 output rows
        // (each counted in by the warps that stored it; see moe_sel.h).  Everything read below was complete before the FFN stored
        // those rows, and the FFN no longer reads this token's x once they are.  Bounded like every wait of this library.
        if (tid <= topk) {
            const unsigned *c = rowcnt + t * (topk + 1) + tid;
            const uint64_t t0 = global_ns();
            while (ld_acquire_gpu(c) < MOE_FFN_ROW_DONE(D)) {
                __nanosleep(100);
                if (global_ns() - t0 > 2000000000ull) {
                    set_status(status, ST_PEER_TIMEOUT | 32);
                    break;
                }
            }
        }
        __syncthreads();
    } else {
        pdl_wait();
    }
    if (nranks > 1) ep_wait(flags, seq, nranks, status);
    float wk[MOE_MAXK], pv[MOE_MAXK];
    const float *wr = &ms->w[0][0] + t * (MOE_MAXK + 1);  // (moe_sel and moe_sel_wide keep w in the same place)
#pragma unroll
    for (uint32_t s = 0; s < MOE_MAXK; s++) wk[s] = s <= topk ? wr[s] : 0.f;
#pragma unroll
    for (uint32_t s = 0; s < MOE_MAXK; s++) pv[s] = s <= topk ? __ldcg(Pg + ((size_t)t * (topk + 1) + s) * D + d) : 0.f;
    float v = h[(size_t)t * D + d];
    float o = 0.f;
#pragma unroll
    for (uint32_t s = 0; s < MOE_MAXK; s++)
        if (s <= topk) o = fmaf(wk[s], pv[s], o);  // rank order, as moe_cmb
    v += __half2float(__float2half_rn(o));
    h[(size_t)t * D + d] = v;
    const float ss = warp_sum(v * v);
    if (lane == 0) tmp[warp] = ss;
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < 8) {  // thread r pushes this block's partial sum into block r's array: after the one cluster barrier nobody touches another block's memory
        float b = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) b += tmp[i];
        *cl.map_shared_rank(&parts[blockIdx.x & 7], tid) = b;
    }
    cl.sync();
    float tot = 0.f;
#pragma unroll
    for (unsigned r = 0; r < 8; r++) tot += parts[r];
    x[(size_t)t * D + d] = __float2half_rn(v * rsqrtf(tot / D + 1e-6f) * wd);
    if (rowcnt) {
        pdl_wait();  // this kernel's completion must imply the FFN's: later kernels rely on the chain of completed predecessors
        if ((blockIdx.x & 7) == 0 && tid <= topk) rowcnt[t * (topk + 1) + tid] = 0;  // cleared for the next layer's launch
    }
}
// The same for the many rows of a prompt's piece: a block per token, four columns per thread by 16-byte loads.  (Rows fill the device by themselves; the cluster's
// one 4-byte load per row of Pg and thread got 2.9 TB/s, 1024 tokens 38.5 -> 25.8 us.)  Every sum in the cluster form's order: the butterfly of 32 columns runs over eight
// threads and then inside them, eight of those make a 256-column part, eight parts the row.  grid nb x 512
__global__ void __launch_bounds__(512) cmb_rmsnorm_rows_k(float *h, const float *w, __half *x, const moe_sel *ms, const float *Pg, uint32_t topk) {
    constexpr uint32_t D = 2048;
    __shared__ float tmp[64];
    const uint32_t t = blockIdx.x, tid = threadIdx.x;
    pdl_launch();
    const float4 wd = ((const float4 *)w)[tid];  // the norm weights are static
    pdl_wait();
    const float *wr = &ms->w[0][0] + t * (MOE_MAXK + 1);  // (moe_sel and moe_sel_wide keep w in the same place)
    float4 v = ((const float4 *)(h + (size_t)t * D))[tid], o = make_float4(0.f, 0.f, 0.f, 0.f), pv[MOE_MAXK];
#pragma unroll
    for (uint32_t s = 0; s < MOE_MAXK; s++)
        if (s <= topk) pv[s] = __ldcg((const float4 *)(Pg + ((size_t)t * (topk + 1) + s) * D) + tid);
#pragma unroll
    for (uint32_t s = 0; s < MOE_MAXK; s++)
        if (s <= topk) {  // rank order, as moe_cmb
            const float k = wr[s];
            o.x = fmaf(k, pv[s].x, o.x); o.y = fmaf(k, pv[s].y, o.y); o.z = fmaf(k, pv[s].z, o.z); o.w = fmaf(k, pv[s].w, o.w);
        }
    v.x += __half2float(__float2half_rn(o.x)); v.y += __half2float(__float2half_rn(o.y));
    v.z += __half2float(__float2half_rn(o.z)); v.w += __half2float(__float2half_rn(o.w));
    ((float4 *)(h + (size_t)t * D))[tid] = v;
    float4 q = make_float4(v.x * v.x, v.y * v.y, v.z * v.z, v.w * v.w);
#pragma unroll
    for (int off = 4; off; off >>= 1) {  // columns 16, 8 and 4 apart
        q.x += __shfl_xor_sync(0xffffffffu, q.x, off);
        q.y += __shfl_xor_sync(0xffffffffu, q.y, off);
        q.z += __shfl_xor_sync(0xffffffffu, q.z, off);
        q.w += __shfl_xor_sync(0xffffffffu, q.w, off);
    }
    const float ss = (q.x + q.z) + (q.y + q.w);  // 2 and 1 apart
    if ((tid & 7) == 0) tmp[tid >> 3] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        float b = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) b += tmp[8 * r + i];
        tot += b;
    }
    const float r = rsqrtf(tot / D + 1e-6f);
    const __half2 lo = __halves2half2(__float2half_rn(v.x * r * wd.x), __float2half_rn(v.y * r * wd.y)), hi = __halves2half2(__float2half_rn(v.z * r * wd.z), __float2half_rn(v.w * r * wd.w));
    ((uint2 *)(x + (size_t)t * D))[tid] = make_uint2(*(const uint32_t *)&lo, *(const uint32_t *)&hi);
}
static cudaError_t launch_add_rmsnorm(const QwLaunch &L) {
    struct { uint32_t nb, D; } a = L.bytes<decltype(a)>(4);
    QW_CHECK_ARG(L.buf<void>(0) && L.buf<void>(2) && L.buf<void>(3) && L.has_bytes(4, 8) && a.nb >= 1 && a.nb <= (uint32_t)L.def("ROWS", 64));
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * a.D * 4 && L.avail(2) >= (size_t)a.D * 4 && L.avail(3) >= (size_t)a.nb * a.D * 2);
    if (L.def("CMB", 0)) {
        const uint32_t topk = (uint32_t)L.def("TOPK", 10);
        const bool wide = L.def("WIDE", 0) != 0;
        QW_CHECK_ARG(a.nb <= (wide ? MOE_MAXB_WIDE : MOE_MAXB));
        QW_CHECK_ARG(L.buf<void>(5) && L.buf<void>(6) && L.avail(5) >= (wide ? sizeof(moe_sel_wide) : sizeof(moe_sel)) && L.avail(6) >= (size_t)a.nb * (topk + 1) * a.D * 4 && topk < MOE_MAXK);
        // EPX = number of expert-parallel ranks whose down projections store into Pg: 7 = this rank's flag array
        // (one sequence number per rank), 8 = this rank's sequence counter
        const uint32_t nranks = (uint32_t)L.def("EPX", 1);
        if (nranks > 1) QW_CHECK_ARG(nranks <= 8 && L.buf<void>(7) && L.avail(7) >= nranks * 4 && L.buf<void>(8) && L.avail(8) >= 4);
        if (a.D == 2048) {
            // ROWCNT defined 1 (one GPU, after moe_ffn): 9 = the FFN's scratch buffer, whose per-row counters replace the wait for the launch
            unsigned *rowcnt = nullptr;
            if (L.def("ROWCNT", 0)) {
                QW_CHECK_ARG(nranks == 1 && !wide && L.buf<unsigned>(9) && L.avail(9) >= MOE_FFN_SYNC_BYTES);
                rowcnt = L.buf<unsigned>(9) + MOE_FFN_ROWCNT;
            }
            // many rows by 16-byte loads; buffers that do not lie at such boundaries (the engine's do) go through the cluster form, whose loads are of 4 bytes
            if (wide && a.nb > MOE_MAXB && nranks == 1 && (((uintptr_t)L.buf<void>(0) | (uintptr_t)L.buf<void>(2) | (uintptr_t)L.buf<void>(3) | (uintptr_t)L.buf<void>(6)) & 15) == 0) {
                qw_launch(cmb_rmsnorm_rows_k, a.nb, 512, 0, L.stream, L.buf<float>(0), L.buf<float>(2), L.buf<__half>(3), L.buf<moe_sel>(5), L.buf<float>(6), topk);
                return cudaGetLastError();
            }
            qw_launch(cmb_rmsnorm_cl_k, a.nb * 8, 256, 0, L.stream, L.buf<float>(0), L.buf<float>(2), L.buf<__half>(3), L.buf<moe_sel>(5), L.buf<float>(6), topk,
                      nranks > 1 ? L.buf<unsigned>(7) : nullptr, nranks > 1 ? L.buf<unsigned>(8) : nullptr, nranks, rowcnt, (unsigned *)L.status);
            return cudaGetLastError();
        }
        qw_launch(add_rmsnorm_k<2>, a.nb, 1024, 0, L.stream, L.buf<float>(0), nullptr, L.buf<float>(2), L.buf<__half>(3), a.D, L.buf<moe_sel>(5), L.buf<float>(6), topk,
                  nranks > 1 ? L.buf<unsigned>(7) : nullptr, nranks > 1 ? L.buf<unsigned>(8) : nullptr, nranks, (unsigned *)L.status);
    } else if (L.def("ADD", 0)) {
        QW_CHECK_ARG(L.buf<void>(1) && L.avail(1) >= (size_t)a.nb * a.D * 2);
        const uint32_t nranks = (uint32_t)L.def("EPX", 1);  // the delta rows were stored by the ranks that own the slots: same binds 7, 8
        if (nranks > 1) QW_CHECK_ARG(nranks <= 8 && L.buf<void>(7) && L.avail(7) >= nranks * 4 && L.buf<void>(8) && L.avail(8) >= 4);
        qw_launch(add_rmsnorm_k<1>, a.nb, 512, 0, L.stream, L.buf<float>(0), L.buf<__half>(1), L.buf<float>(2), L.buf<__half>(3), a.D, nullptr, nullptr, 0,
                  nranks > 1 ? L.buf<unsigned>(7) : nullptr, nranks > 1 ? L.buf<unsigned>(8) : nullptr, nranks, (unsigned *)L.status);
    } else {
        qw_launch(add_rmsnorm_k<0>, a.nb, 512, 0, L.stream, L.buf<float>(0), nullptr, L.buf<float>(2), L.buf<__half>(3), a.D, nullptr, nullptr, 0, nullptr, nullptr, 1, nullptr);
    }
    return cudaGetLastError();
}
QW_FAMILY(add_rmsnorm, launch_add_rmsnorm, 256)

// A rank that has no row to contribute to an exchange still has to publish its sequence number.
// binds: 11 = {seq, done} counters, 12 = {rank}, 24 + r = flag array of rank r; define EPX = number of ranks.  grid 1 x 32
__global__ void ep_publish_k(const EpPeers ep) {
    pdl_sync();
    ep_publish(ep);
}
static cudaError_t launch_ep_publish(const QwLaunch &L) {
    EpPeers ep{};
    ep.nranks = (uint32_t)L.def("EPX", 0);
    QW_CHECK_ARG(ep.nranks >= 2 && ep.nranks <= 8 && L.has_bytes(12, 4) && L.buf<unsigned>(11) && L.avail(11) >= 8);
    ep.rank = L.bytes<uint32_t>(12);
    QW_CHECK_ARG(ep.rank < ep.nranks);
    ep.seq = L.buf<unsigned>(11);
    ep.done = ep.seq + 1;
    for (uint32_t r = 0; r < ep.nranks; r++) {
        ep.flagR[r] = L.buf<unsigned>(24 + r);
        QW_CHECK_ARG(ep.flagR[r] && L.avail(24 + r) >= ep.nranks * 4);
    }
    qw_launch(ep_publish_k, 1, 32, 0, L.stream, ep);
    return cudaGetLastError();
}
QW_FAMILY(ep_publish, launch_ep_publish, 32)

// binds: 0 = logits fp32 [nb][V], 1 = ids out int32 [nb], 2 = {nb, V}, 3 = second ids out (with IDS2 defined 1,
// e.g. a host-visible copy).  With ALT defined 1 also 4 = a position: with an odd one the second ids go 64 places further, so that the
// host can read a step's while the next step runs.  grid nb x 1024
__global__ void __launch_bounds__(1024) k_argmax_k(const float *lg, int32_t *ids, int32_t *ids2, uint32_t V, const int32_t *pos) {
    __shared__ float bv[32];
    __shared__ uint32_t bi[32];
    pdl_sync();
    const uint32_t t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *r = lg + (size_t)t * V;
    float best = -INFINITY;
    uint32_t idx = 0xffffffffu;
    for (uint32_t i = tid; i < V; i += 1024) {
        const float v = r[i];
        if (v > best || idx == 0xffffffffu) { best = v; idx = i; }  // strictly greater: the lowest index of equals stays
    }
    auto better = [](float v, uint32_t i, float bv2, uint32_t bi2) { return v > bv2 || (v == bv2 && i < bi2); };
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, off);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, off);
        if (better(ov, oi, best, idx)) { best = ov; idx = oi; }
    }
    if (lane == 0) { bv[warp] = best; bi[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        best = bv[lane];
        idx = bi[lane];
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, off);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, off);
            if (better(ov, oi, best, idx)) { best = ov; idx = oi; }
        }
        if (lane == 0) {
            ids[t] = (int32_t)idx;
            if (ids2) ids2[t + (pos ? (*pos & 1) * 64 : 0)] = (int32_t)idx;
        }
    }
}
static cudaError_t launch_k_argmax(const QwLaunch &L) {
    struct { uint32_t nb, V; } a = L.bytes<decltype(a)>(2);
    QW_CHECK_ARG(L.buf<void>(0) && L.buf<void>(1) && L.has_bytes(2, 8) && a.nb >= 1 && a.nb <= 64 && a.V >= 1);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * a.V * 4 && L.avail(1) >= a.nb * 4);
    int32_t *ids2 = L.def("IDS2", 0) ? L.buf<int32_t>(3) : nullptr;
    const bool alt = ids2 && L.def("ALT", 0);
    const int32_t *pos = alt ? L.buf<int32_t>(4) : nullptr;
    if (L.def("IDS2", 0)) QW_CHECK_ARG(ids2 && L.avail(3) >= (alt ? 64 + a.nb : a.nb) * 4 && (!alt || (pos && L.avail(4) >= 4)));
    qw_launch(k_argmax_k, a.nb, 1024, 0, L.stream, L.buf<float>(0), L.buf<int32_t>(1), ids2, a.V, pos);
    return cudaGetLastError();
}
QW_FAMILY(k_argmax, launch_k_argmax, 1024)

// binds: 0 = pos int32 [nb], 3 = {nb}; with FEED defined 1 also 1 = tok int32 [nb], 2 = sampled ids int32 [nb]
__global__ void par_advance_k(int32_t *pos, int32_t *tok, const int32_t *ids, uint32_t nb) {
    pdl_sync();
    const uint32_t t = threadIdx.x;
    if (t >= nb) return;
    pos[t] += 1;
    if (tok && ids) tok[t] = ids[t];
}
static cudaError_t launch_par_advance(const QwLaunch &L) {
    const uint32_t nb = L.bytes<uint32_t>(3);
    QW_CHECK_ARG(L.buf<void>(0) && nb >= 1 && nb <= 64 && L.avail(0) >= nb * 4);
    const bool feed = L.def("FEED", 0) != 0;
    if (feed) QW_CHECK_ARG(L.buf<void>(1) && L.buf<void>(2) && L.avail(1) >= nb * 4 && L.avail(2) >= nb * 4);
    qw_launch(par_advance_k, 1, 64, 0, L.stream, L.buf<int32_t>(0), feed ? L.buf<int32_t>(1) : nullptr, feed ? L.buf<int32_t>(2) : nullptr, nb);
    return cudaGetLastError();
}
QW_FAMILY(par_advance, launch_par_advance, 64)

// The step's control block (token, slot id, position per row) is written by the host into pinned memory; this
// copies it into device memory once so that no other kernel reads across PCIe.
// binds: 0 = source int32, 1 = destination int32, 2 = {count}
__global__ void par_begin_k(const int32_t *src, int32_t *dst, uint32_t n) {
    pdl_sync();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}
static cudaError_t launch_par_begin(const QwLaunch &L) {
    const uint32_t n = L.bytes<uint32_t>(2);
    QW_CHECK_ARG(L.buf<void>(0) && L.buf<void>(1) && n >= 1 && L.avail(0) >= n * 4 && L.avail(1) >= n * 4);
    qw_launch(par_begin_k, 1, 256, 0, L.stream, L.buf<int32_t>(0), L.buf<int32_t>(1), n);
    return cudaGetLastError();
}
QW_FAMILY(par_begin, launch_par_begin, 256)

// Control block of a piece of a prompt: n consecutive tokens of one slot, newest first (row r = prompt position p0 + n - 1 - r), so
// that the piece's last token is row 0.  The prompt was copied to the device once; nothing is read from the host per piece.
// binds: 0 = prompt int32, 1 = control block [3][rows] (token, slot, position), 2 = {p0, n, slot, rows}
struct par_chunk_args { uint32_t p0, n, slot, rows; };
__global__ void par_chunk_k(const int32_t *prompt, int32_t *ctl, par_chunk_args a) {
    pdl_sync();
    for (uint32_t r = threadIdx.x; r < a.n; r += blockDim.x) {
        const uint32_t pos = a.p0 + a.n - 1 - r;
        ctl[r] = prompt[pos];
        ctl[a.rows + r] = (int32_t)a.slot;
        ctl[2 * a.rows + r] = (int32_t)pos;
    }
}
static cudaError_t launch_par_chunk(const QwLaunch &L) {
    const par_chunk_args a = L.bytes<par_chunk_args>(2);
    QW_CHECK_ARG(L.has_bytes(2, 16) && L.buf<void>(0) && L.buf<void>(1) && a.n >= 1 && a.n <= a.rows && L.avail(0) >= ((size_t)a.p0 + a.n) * 4 &&
                 L.avail(1) >= (size_t)a.rows * 12);
    qw_launch(par_chunk_k, 1, 256, 0, L.stream, L.buf<int32_t>(0), L.buf<int32_t>(1), a);
    return cudaGetLastError();
}
QW_FAMILY(par_chunk, launch_par_chunk, 256)

// ------------------------------------------------------------------------------------------------ fill
// Counter-based generator: byte i of a tensor with seed s is the low byte of mix64(s * 0x9E3779B97F4A7C15 + i)
// (qwental_b200/synth.py holds the same functions in numpy).
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t hash_u64(uint64_t seed, uint64_t i) { return mix64(seed * 0x9E3779B97F4A7C15ull + i); }

struct fill_args {
    uint64_t seed, count;  // count: bytes (modes 0-2), elements (modes 3-5)
    uint64_t base;         // index of the first byte / element within the whole tensor (a rank's slice of a sharded tensor)
    uint32_t mode;         // 0 zero bytes, 1 IQ3_S blocks, 2 Q8_0 blocks, 3 fp16 normal, 4 fp32 normal, 5 fp32 constant
    float p0;              // multiplier of the block scale d (modes 1, 2), std (modes 3, 4) or the constant (mode 5)
    float p1;              // mean added (modes 3, 4)
};

__device__ __forceinline__ float hash_normal(uint64_t seed, uint64_t i) {
    const uint64_t h = hash_u64(seed, i);
    const float u1 = ((float)(uint32_t)(h >> 40) + 1.0f) * (1.0f / 16777216.0f);
    const float u2 = (float)(uint32_t)((h >> 16) & 0xFFFFFF) * (1.0f / 16777216.0f);
    return sqrtf(-2.0f * logf(u1)) * cosf(6.283185307179586f * u2);
}

__global__ void qw_fill_k(uint8_t *dst, fill_args a) {
    pdl_sync();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    if (a.mode == 0 && (((uintptr_t)dst | a.count) & 15) == 0) {  // zeroing: 16 bytes per store
        for (uint64_t li = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; li < a.count / 16; li += stride) ((uint4 *)dst)[li] = make_uint4(0, 0, 0, 0);
        return;
    }
    for (uint64_t li = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; li < a.count; li += stride) {
        const uint64_t i = a.base + li;
        if (a.mode == 0) dst[li] = 0;
        else if (a.mode == 1 || a.mode == 2) {
            const uint32_t bb = a.mode == 1 ? 110 : 34;
            const uint64_t blk = i / bb;
            const uint32_t off = (uint32_t)(i % bb);
            uint8_t by = (uint8_t)(hash_u64(a.seed, i) & 0xFF);
            if (a.mode == 2 && by == 0x80) by = 0x81;
            if (off < 2) {
                const float u = (float)(uint32_t)(hash_u64(a.seed ^ 0x5CA1Eull, blk) >> 40) * (1.0f / 16777216.0f);
                const float d = __fmul_rn(__fadd_rn(1e-3f, __fmul_rn(u, 1.9e-2f)), a.p0);
                const uint16_t hb = __half_as_ushort(__float2half_rn(d));
                by = off == 0 ? (uint8_t)(hb & 0xFF) : (uint8_t)(hb >> 8);
            }
            dst[li] = by;
        } else if (a.mode == 3) ((__half *)dst)[li] = __float2half_rn(hash_normal(a.seed, i) * a.p0 + a.p1);
        else if (a.mode == 4) ((float *)dst)[li] = hash_normal(a.seed, i) * a.p0 + a.p1;
        else ((float *)dst)[li] = a.p0;
    }
}
// binds: 0 = destination, 1 = fill_args
static cudaError_t launch_qw_fill(const QwLaunch &L) {
    fill_args a = L.bytes<fill_args>(1);
    QW_CHECK_ARG(L.buf<void>(0) && L.has_bytes(1, 36) && a.mode <= 5 && a.count > 0);
    const size_t esz = a.mode <= 2 ? 1 : a.mode == 3 ? 2 : 4;
    QW_CHECK_ARG(L.avail(0) >= a.count * esz);
    const uint64_t blocks = ((a.mode == 0 ? a.count / 16 : a.count) + 255) / 256 + 1;
    const unsigned grid = (unsigned)(blocks < (uint64_t)L.sm_count * 32 ? blocks : (uint64_t)L.sm_count * 32);
    qw_launch(qw_fill_k, grid, 256, 0, L.stream, L.buf<uint8_t>(0), a);
    return cudaGetLastError();
}
QW_FAMILY(qw_fill, launch_qw_fill, 256)
