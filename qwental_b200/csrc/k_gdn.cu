// Gated DeltaNet decode step for all slots in one launch, with each slot's fp32 state resident in HBM.
//
//   dn_epi     epilogue of the GDN input projection: depthwise conv-4 + SiLU with the slot's own conv state,
//              a -> log-decay A_neg*softplus(a + dt_bias), b -> beta = sigmoid(b)
//              -- role of dn_epi_rowT, kernels/dn_proj.metal:190-244 (the projection itself is qmv_mma; the
//                 reference rounds the projection to fp16 before this epilogue, :199, so nothing is lost)
//   gdn_fstep  L2-norm of q and k, S <- g*S; mem = S^T k; delta = beta*(v - mem); S += k delta^T; o = S^T q,
//              then the gated RMSNorm o*rsqrt(mean o^2 + eps)*w*sigmoid(z)
//              -- role of gdn_fstep, kernels/gdn_decode.metal:299-418 (q/k norm :281-296)
//
// The reference launches gdn_fstep once per slot (src/engine.c:8992-9007); here the slot is a grid dimension
// and the per-slot state is found through a slot-id table, so the launch count does not grow with the batch.
// A slot's arithmetic never looks at another slot, so batched results equal the slot alone bit for bit.
#include "common.cuh"
#include "qw_kern.h"

using namespace qw;

#define GDN_EPS 1e-6f
#define GDN_SEQ_MAX 1024  // tokens of one launch of the sequence kernels
#define GDN_SEQ_CHUNK 16  // tokens of one of gdn_seq's two staging buffers

// proj row layout (fp16, stride PS): [q: HK*DK | k: HK*DK | v: HV*DV | z: HV*DV | a: HV | b: HV]
struct dn_epi_args {
    uint32_t nb, layer, nlayers, proj_stride;
};

// The epilogue of a channel, shared by the forms below so that they give the same bits.  (The multiply-adds of the convolution are spelt out: left to
// the compiler, the sum may be contracted in one way in one kernel and in another way in the next.)  s3 = the newest of the channel's last four inputs
__device__ __forceinline__ __half dn_conv(const float4 &w, float s0, float s1, float s2, float s3) {
    const float y = __fmaf_rn(w.w, s3, __fmaf_rn(w.z, s2, __fmaf_rn(w.x, s0, __fmul_rn(w.y, s1))));
    return __float2half_rn(y / (1.0f + expf(-y)));
}
__device__ __forceinline__ float dn_decay(float a, float dtb, float An) {
    const float xa = a + dtb;
    const float sp = xa > 20.0f ? xa : logf(1.0f + expf(xa));
    return An * sp;
}
__device__ __forceinline__ float dn_beta(float b) { return 1.0f / (1.0f + expf(-b)); }

// binds: 0 = proj fp16 [nb][proj_stride], 1 = conv weights fp32 [C][4], 2 = conv state pool fp32
// [slot][nlayers][3][C], 3 = A_neg fp32 [HV], 4 = dt_bias fp32 [HV], 5 = cv out fp16 [nb][C],
// 6 = la fp32 [nb][HV], 7 = beta fp32 [nb][HV], 8 = slot ids int32 [nb], 9 = dn_epi_args.
// grid (ceil((C + 2 HV)/256), nb) x 256
__global__ void __launch_bounds__(256) dn_epi_k(const __half *proj, const float *cw, float *pool, const float *An, const float *dtb, __half *cv,
                                               float *la, float *be, const int32_t *sids, dn_epi_args a, uint32_t C, uint32_t HV, bool early) {
    pdl_launch();
    if (!early) pdl_wait();
    const uint32_t g = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
    const __half *pr = proj + (size_t)t * a.proj_stride;
    if (g < C) {
        // early: the slot table, the conv state and the static weights are read before the wait for the projection (see gdn_fstep_k for
        // when that is allowed)
        float *st = pool + ((size_t)sids[t] * a.nlayers + a.layer) * 3 * C;
        const float s0 = st[g], s1 = st[C + g], s2 = st[2 * C + g];
        const float4 w = *(const float4 *)(cw + 4 * (size_t)g);
        if (early) pdl_wait();
        const float s3 = __half2float(pr[g]);
        cv[(size_t)t * C + g] = dn_conv(w, s0, s1, s2, s3);
        st[g] = s1;
        st[C + g] = s2;
        st[2 * C + g] = s3;
    } else if (g < C + HV) {
        if (early) pdl_wait();
        const uint32_t j = g - C;
        la[t * HV + j] = dn_decay(__half2float(pr[C + HV * 128 + j]), dtb[j], An[j]);
    } else if (g < C + 2 * HV) {
        if (early) pdl_wait();
        const uint32_t j = g - C - HV;
        be[t * HV + j] = dn_beta(__half2float(pr[C + HV * 128 + HV + j]));
    }
}

static cudaError_t launch_dn_epi(const QwLaunch &L) {
    const uint32_t HK = (uint32_t)L.def("HK", 16), HV = (uint32_t)L.def("HV", 32), DK = (uint32_t)L.def("DK", 128), DV = (uint32_t)L.def("DV", 128);
    const uint32_t C = 2 * HK * DK + HV * DV;
    dn_epi_args a = L.bytes<dn_epi_args>(9);
    QW_CHECK_ARG(DV == 128 && DK == 128 && L.has_bytes(9, 16) && a.nb >= 1 && a.nb <= 64 && a.layer < a.nlayers);
    QW_CHECK_ARG(a.proj_stride >= C + HV * DV + 2 * HV);
    for (int i = 0; i <= 8; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= ((size_t)(a.nb - 1) * a.proj_stride + C + HV * DV + 2 * HV) * 2 && L.avail(1) >= (size_t)C * 16 &&
                 L.avail(5) >= (size_t)a.nb * C * 2 && L.avail(6) >= (size_t)a.nb * HV * 4 && L.avail(7) >= (size_t)a.nb * HV * 4 &&
                 L.avail(8) >= (size_t)a.nb * 4);
    qw_launch(dn_epi_k, dim3((C + 2 * HV + 255) / 256, a.nb), 256, 0, L.stream, L.buf<__half>(0), L.buf<float>(1), L.buf<float>(2), L.buf<float>(3),
                                                                        L.buf<float>(4), L.buf<__half>(5), L.buf<float>(6), L.buf<float>(7),
                                                                        L.buf<int32_t>(8), a, C, HV, L.def("EARLY", 0) != 0);
    return cudaGetLastError();
}
QW_FAMILY(dn_epi, launch_dn_epi, 256)

// The same epilogue for nb consecutive tokens of ONE slot (a piece of a prompt), newest token first: row r is the token at
// sequence position nb - 1 - r of the piece.  A token's three predecessors are rows of the same projection (the state holds
// exactly those fp16 values as fp32) or, for the first three tokens, the slot's conv state, which this kernel only reads:
// gdn_seq, the next launch, writes the piece's last three inputs into it.
// A thread takes V channels of RUN consecutive tokens.  More than 64 tokens: eight channels as 16 bytes of two tokens, whose inputs slide through the window
// (419 tokens on a B200: 21.9 -> 15.9 us); fewer want every channel of a token on a thread of its own (45 tokens: 5.9, the other form 6.7).  The last block of a row
// of blocks does decay and beta.
// binds as dn_epi (2 is not written).  grid (ceil(C / (128 V)) + 1, ceil(nb / RUN)) x 128
template <int V>
__device__ __forceinline__ void load_halves(const __half *p, float (&f)[V]) {
    if constexpr (V == 8) {
        const uint4 v = *(const uint4 *)p;
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 x = __half22float2(*(const __half2 *)&w[i]);
            f[2 * i] = x.x;
            f[2 * i + 1] = x.y;
        }
    } else f[0] = __half2float(p[0]);
}
template <int V, uint32_t RUN>
__global__ void __launch_bounds__(128) dn_epi_seq_k(const __half *proj, const float *cw, const float *pool, const float *An, const float *dtb, __half *cv,
                                                    float *la, float *be, const int32_t *sids, dn_epi_args a, uint32_t C, uint32_t HV) {
    pdl_launch();
    const uint32_t tau0 = blockIdx.y * RUN, tau1 = tau0 + RUN < a.nb ? tau0 + RUN : a.nb;  // positions in the piece: row nb - 1 - tau
    if (blockIdx.x == gridDim.x - 1) {
        pdl_wait();
        for (uint32_t i = threadIdx.x; i < (tau1 - tau0) * 2 * HV; i += 128) {
            const uint32_t t = a.nb - 1 - (tau0 + i / (2 * HV)), j = i % (2 * HV);
            const float v = __half2float(proj[(size_t)t * a.proj_stride + C + HV * 128 + j]);
            if (j < HV) la[t * HV + j] = dn_decay(v, dtb[j], An[j]);
            else be[t * HV + j - HV] = dn_beta(v);
        }
        return;
    }
    const uint32_t g = (blockIdx.x * 128 + threadIdx.x) * V;
    float4 w[V];
    if (g < C)
#pragma unroll
        for (int i = 0; i < V; i++) w[i] = *(const float4 *)(cw + 4 * (size_t)(g + i));
    pdl_wait();
    if (g >= C) return;
    const float *st = pool + ((size_t)sids[0] * a.nlayers + a.layer) * 3 * C + g;
    const __half *last = proj + (size_t)(a.nb - 1) * a.proj_stride + g;  // position 0; position tau is tau rows before it
    float s[3][V];  // the three inputs before the run
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int tau = (int)tau0 - 3 + k;
        if (tau >= 0) load_halves<V>(last - (size_t)tau * a.proj_stride, s[k]);
        else
#pragma unroll
            for (int i = 0; i < V; i++) s[k][i] = st[(size_t)(3 + tau) * C + i];
    }
#pragma unroll
    for (uint32_t n = 0; n < RUN; n++) {
        const uint32_t tau = tau0 + n;
        if (tau >= tau1) break;
        float x[V];
        load_halves<V>(last - (size_t)tau * a.proj_stride, x);
        __half o[V];
#pragma unroll
        for (int i = 0; i < V; i++) {
            o[i] = dn_conv(w[i], s[0][i], s[1][i], s[2][i], x[i]);
            s[0][i] = s[1][i];
            s[1][i] = s[2][i];
            s[2][i] = x[i];
        }
        __half *out = cv + (size_t)(a.nb - 1 - tau) * C + g;
        if constexpr (V == 8) {
            uint32_t u[4];
#pragma unroll
            for (int i = 0; i < 4; i++) u[i] = (uint32_t)__half_as_ushort(o[2 * i]) | (uint32_t)__half_as_ushort(o[2 * i + 1]) << 16;
            *(uint4 *)out = make_uint4(u[0], u[1], u[2], u[3]);
        } else out[0] = o[0];
    }
}

static cudaError_t launch_dn_epi_seq(const QwLaunch &L) {
    const uint32_t HK = (uint32_t)L.def("HK", 16), HV = (uint32_t)L.def("HV", 32), DK = (uint32_t)L.def("DK", 128), DV = (uint32_t)L.def("DV", 128);
    const uint32_t C = 2 * HK * DK + HV * DV;
    dn_epi_args a = L.bytes<dn_epi_args>(9);
    QW_CHECK_ARG(DV == 128 && DK == 128 && L.has_bytes(9, 16) && a.nb >= 1 && a.nb <= GDN_SEQ_MAX && a.layer < a.nlayers);
    QW_CHECK_ARG(a.proj_stride >= C + HV * DV + 2 * HV);
    for (int i = 0; i <= 8; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= ((size_t)(a.nb - 1) * a.proj_stride + C + HV * DV + 2 * HV) * 2 && L.avail(1) >= (size_t)C * 16 &&
                 L.avail(5) >= (size_t)a.nb * C * 2 && L.avail(6) >= (size_t)a.nb * HV * 4 && L.avail(7) >= (size_t)a.nb * HV * 4 && L.avail(8) >= 4);
    // (C is a multiple of 128)
    const bool vec = a.nb > 64 && a.proj_stride % 8 == 0 && (((uintptr_t)L.buf<void>(0) | (uintptr_t)L.buf<void>(5)) & 15) == 0;
    qw_launch(vec ? dn_epi_seq_k<8, 2> : dn_epi_seq_k<1, 1>, dim3((C + (vec ? 1023 : 127)) / (vec ? 1024 : 128) + 1, vec ? (a.nb + 1) / 2 : a.nb), 128, 0, L.stream, L.buf<__half>(0),
              L.buf<float>(1), L.buf<float>(2), L.buf<float>(3), L.buf<float>(4), L.buf<__half>(5), L.buf<float>(6), L.buf<float>(7), L.buf<int32_t>(8), a, C, HV);
    return cudaGetLastError();
}
QW_FAMILY(dn_epi_seq, launch_dn_epi_seq, 256)

// ------------------------------------------------------------------------------------------------ recurrent step
struct gdn_args {
    uint32_t nb, layer, nlayers, z_stride;  // z: fp16 rows of stride z_stride (the z part of the projection)
};

// One block per (v-head, slot): 512 threads, thread (rq = tid / 32, c4 = tid % 32) holds rows 8 rq .. 8 rq + 7 of columns
// 4 c4 .. 4 c4 + 3 of the head's [DK][DV] state in registers: every state access is a 16-byte load or store and a warp
// moves one whole 512-byte row per instruction.  The 16 row groups meet in shared memory (summed in group order); q and k
// are normalised by every warp for itself, so the block has three barriers in all.
// binds: 0 = cv fp16 [nb][C], 1 = la [nb][HV], 2 = beta [nb][HV], 3 = state pool fp32 [slot][nlayers][HV][DK][DV],
// 4 = z fp16, 5 = norm weight fp32 [DV], 6 = gy out fp16 [nb][HV*DV], 7 = slot ids, 8 = gdn_args; with O_OUT
// defined 1 also 9 = o out fp16 [nb][HV*DV] (the un-normalised output, for tests).  grid (HV, nb) x 512
template <bool TILED>
__global__ void __launch_bounds__(512, 2) gdn_fstep_k(const __half *cv, const float *la, const float *beta, float *pool, const __half *z,
                                                  const float *nw, __half *gy, const int32_t *sids, __half *oo, gdn_args a, uint32_t HK, uint32_t HV,
                                                  bool early) {
    constexpr int DK = 128, DV = 128;
    __shared__ float red[8];
    __shared__ float4 part[2][16][32];  // [S^T k | S^T q][row group][column quad]
    pdl_launch();
    if (!early) pdl_wait();
    const uint32_t hv = blockIdx.x, t = blockIdx.y, tid = threadIdx.x, c4 = tid & 31, rq = tid >> 5, lane = tid & 31, warp = tid >> 5;
    const uint32_t hk = TILED ? hv % HK : hv / (HV / HK);
    const uint32_t C = 2 * HK * DK + HV * DV;
    const __half *row = cv + (size_t)t * C;
    float4 *S = (float4 *)(pool + (((size_t)sids[t] * a.nlayers + a.layer) * HV + hv) * DK * DV) + c4;

    // State rows into registers: the long-latency part.  With EARLY defined 1 they, and the slot id they are found by, are requested before the
    // wait for the previous kernel.  The state was last written a step earlier, which may still be running; the slot table by
    // par_begin at the start of this step, possibly.  A launch cannot begin before every block of its predecessor has started, but that alone says
    // little: the small launches of a layer can all be resident while par_begin still reads the host's memory.  So the host runs this form
    // only behind two launches that fill every SM (moe_ffn: as many blocks as fit the device) after either writer -- a step has at least three --: the later
    // one cannot have started all its blocks before the earlier one has left, and that one has waited for everything before it.
    float4 s[8];
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = S[(size_t)(8 * rq + i) * (DV / 4)];
    if (early) pdl_wait();  // q, k, v, z, the decay and beta are the previous kernels' output

    // q / k L2 normalisation, by every warp for itself (no block barrier): lane l squares elements 4l .. 4l+3, one butterfly
    // gives the head's sum of squares; then the warp's own eight rows 8 rq .. 8 rq + 7 are scaled
    const __half *qh = row + hk * DK, *kh = row + HK * DK + hk * DK;
    float qn[8], kn[8];
    {
        const uint2 q4 = *(const uint2 *)(qh + 4 * lane), k4 = *(const uint2 *)(kh + 4 * lane);
        const float2 qa = __half22float2(*(const __half2 *)&q4.x), qb = __half22float2(*(const __half2 *)&q4.y);
        const float2 ka = __half22float2(*(const __half2 *)&k4.x), kb = __half22float2(*(const __half2 *)&k4.y);
        const float qss = warp_sum(fmaf(qa.x, qa.x, fmaf(qa.y, qa.y, fmaf(qb.x, qb.x, qb.y * qb.y))));
        const float kss = warp_sum(fmaf(ka.x, ka.x, fmaf(ka.y, ka.y, fmaf(kb.x, kb.x, kb.y * kb.y))));
        const float rq_ = rsqrtf(qss / DK + GDN_EPS), rk_ = rsqrtf(kss / DK + GDN_EPS);
        const uint4 qr = *(const uint4 *)(qh + 8 * rq), kr = *(const uint4 *)(kh + 8 * rq);  // the warp's eight rows (same for all lanes)
        const uint32_t qw[4] = {qr.x, qr.y, qr.z, qr.w}, kw[4] = {kr.x, kr.y, kr.z, kr.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 qf = __half22float2(*(const __half2 *)&qw[j]), kf = __half22float2(*(const __half2 *)&kw[j]);
            qn[2 * j] = __half2float(__float2half_rn(qf.x * rq_ / DK));
            qn[2 * j + 1] = __half2float(__float2half_rn(qf.y * rq_ / DK));
            kn[2 * j] = __half2float(__float2half_rn(kf.x * rk_ * rsqrtf((float)DK)));
            kn[2 * j + 1] = __half2float(__float2half_rn(kf.y * rk_ * rsqrtf((float)DK)));
        }
    }

    const float gdec = expf(la[t * HV + hv]), b = beta[t * HV + hv];
    float4 mem = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float kk = kn[i];
        s[i].x *= gdec; s[i].y *= gdec; s[i].z *= gdec; s[i].w *= gdec;
        mem.x = fmaf(s[i].x, kk, mem.x); mem.y = fmaf(s[i].y, kk, mem.y); mem.z = fmaf(s[i].z, kk, mem.z); mem.w = fmaf(s[i].w, kk, mem.w);
    }
    part[0][rq][c4] = mem;
    __syncthreads();
    mem = part[0][0][c4];
#pragma unroll
    for (int r = 1; r < 16; r++) {
        const float4 pv = part[0][r][c4];
        mem.x += pv.x; mem.y += pv.y; mem.z += pv.z; mem.w += pv.w;
    }
    const uint2 vraw = *(const uint2 *)(row + 2 * HK * DK + hv * DV + 4 * c4);
    const float2 v01 = __half22float2(*(const __half2 *)&vraw.x), v23 = __half22float2(*(const __half2 *)&vraw.y);
    const float4 d = make_float4(b * (v01.x - mem.x), b * (v01.y - mem.y), b * (v23.x - mem.z), b * (v23.y - mem.w));
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float kk = kn[i], qq = qn[i];
        s[i].x = fmaf(kk, d.x, s[i].x); s[i].y = fmaf(kk, d.y, s[i].y); s[i].z = fmaf(kk, d.z, s[i].z); s[i].w = fmaf(kk, d.w, s[i].w);
        out.x = fmaf(s[i].x, qq, out.x); out.y = fmaf(s[i].y, qq, out.y); out.z = fmaf(s[i].z, qq, out.z); out.w = fmaf(s[i].w, qq, out.w);
    }
    part[1][rq][c4] = out;
#pragma unroll
    for (int i = 0; i < 8; i++) S[(size_t)(8 * rq + i) * (DV / 4)] = s[i];
    __syncthreads();
    float o1 = 0.f;
    const uint32_t c = tid;  // threads 0..127: one output column each
    if (tid < 128) {
        const float *pc = (const float *)&part[1][0][0] + c;
        o1 = pc[0];
#pragma unroll
        for (int r = 1; r < 16; r++) o1 += pc[r * 128];
        const __half oh = __float2half_rn(o1);
        if (oo) oo[(size_t)t * HV * DV + hv * DV + c] = oh;
        const float x = __half2float(oh);  // the norm sees the fp16-rounded output (kernels/gdn_decode.metal:386,408)
        const float p = warp_sum(x * x);
        if (lane == 0) red[warp] = p;
    }
    __syncthreads();
    if (tid < 128) {
        const float r = rsqrtf((((red[0] + red[1]) + red[2]) + red[3]) / DV + GDN_EPS);
        const float x = __half2float(__float2half_rn(o1));
        const float zz = __half2float(z[(size_t)t * a.z_stride + hv * DV + c]);
        gy[(size_t)t * HV * DV + hv * DV + c] = __float2half_rn(x * r * nw[c] * (1.0f / (1.0f + expf(-zz))));
    }
}

static cudaError_t launch_gdn_fstep(const QwLaunch &L) {
    const uint32_t HK = (uint32_t)L.def("HK", 16), HV = (uint32_t)L.def("HV", 32), DK = (uint32_t)L.def("DK", 128), DV = (uint32_t)L.def("DV", 128);
    const bool tiled = L.def("GDN_TILED", 1) != 0;
    const uint32_t C = 2 * HK * DK + HV * DV;
    gdn_args a = L.bytes<gdn_args>(8);
    QW_CHECK_ARG(DK == 128 && DV == 128 && HV % HK == 0 && L.has_bytes(8, 16) && a.nb >= 1 && a.nb <= 64 && a.layer < a.nlayers && a.z_stride >= HV * DV);
    for (int i = 0; i <= 7; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * C * 2 && L.avail(1) >= (size_t)a.nb * HV * 4 && L.avail(2) >= (size_t)a.nb * HV * 4 &&
                 L.avail(4) >= ((size_t)(a.nb - 1) * a.z_stride + HV * DV) * 2 && L.avail(5) >= DV * 4 && L.avail(6) >= (size_t)a.nb * HV * DV * 2 &&
                 L.avail(7) >= (size_t)a.nb * 4);
    QW_CHECK_ARG(L.tx == 512);
    const dim3 grid(HV, a.nb);
    const bool early = L.def("EARLY", 0) != 0;
    __half *oo = L.def("O_OUT", 0) ? L.buf<__half>(9) : nullptr;
    if (L.def("O_OUT", 0)) QW_CHECK_ARG(oo && L.avail(9) >= (size_t)a.nb * HV * DV * 2);
    if (tiled)
        qw_launch(gdn_fstep_k<true>, grid, 512, 0, L.stream, L.buf<__half>(0), L.buf<float>(1), L.buf<float>(2), L.buf<float>(3), L.buf<__half>(4),
                                                     L.buf<float>(5), L.buf<__half>(6), L.buf<int32_t>(7), oo, a, HK, HV, early);
    else
        qw_launch(gdn_fstep_k<false>, grid, 512, 0, L.stream, L.buf<__half>(0), L.buf<float>(1), L.buf<float>(2), L.buf<float>(3), L.buf<__half>(4),
                                                      L.buf<float>(5), L.buf<__half>(6), L.buf<int32_t>(7), oo, a, HK, HV, early);
    return cudaGetLastError();
}
QW_FAMILY(gdn_fstep, launch_gdn_fstep, 512)

// ------------------------------------------------------------------------------------------------ recurrence over a piece of a prompt
// nb consecutive tokens of ONE slot (row r = token nb - 1 - r of the piece, as dn_epi_seq): the state is loaded once, the tokens run
// one after another, the state is stored once.  The columns of the state are independent in the recurrence, so a head is split
// over 4 blocks of 32 columns and a block over 4 warps of 8; no block barrier inside the token loop.  A lane holds row groups j and j + 8
// (eight rows each) of two columns as fp32 pairs (row of group j, row of group j + 8): the packed fp32 instructions run both groups' chains at
// once, and an operand read from shared memory serves two columns.  Four more warps work beside them, a buffer ahead and a buffer behind: they
// prepare the next 16 tokens in shared memory (normalised k and q as such pairs, v, decay and beta) and add up the outputs of the last 16.
// Bound by the latency of one token's chain: decay, the fma chain of S^T k, the 16 group sums through shared memory, their ordered sum, the
// update.  Everything else is off it: S^T q of a token runs beside the next token's sums, and its 16 group sums are left to the other warps.
// 419 tokens on a B200: 146 -> 95 us (before, a lane held 32 rows of one column: every fma its own instruction and its own operand from shared
// memory, the running sum handed on by four shuffles); prompts of 419 tokens, 48 layers, 40.3 -> 38.4 ms.  One block per SM, by registers and by shared memory (before, by
// registers alone): 48 and 64 value heads are two waves of 148 blocks, as before; prompts of 1024 tokens, 3 layers, 9.6 -> 5.9 and 11.2 -> 7.0 ms with the rest of the path.
// Bit-identical to nb launches of gdn_fstep: the 16 partial sums of eight rows each are the same fma chains and are added in the same order.
// The gated RMSNorm needs all 128 columns of a head: gdn_gate does it afterwards.
// binds: 0 = cv fp16 [nb][C], 1 = la [nb][HV], 2 = beta [nb][HV], 3 = state pool, 4 = proj fp16 (row stride z_stride), 5 = conv state
// pool (the last three inputs of the piece are written), 6 = o out fp16 [nb][HV*DV] (not normalised), 7 = slot ids (entry 0), 8 = gdn_args.
// grid (4, HV) x 256
// Floats of a staged token: k and q as 8 lane groups of 8 pairs (16 floats, 20 apart: the eight lanes of a 16-byte load read different banks),
// v, then {decay, decay, beta}.  Sums of 16 row groups: a column's 16 floats, 20 apart.
constexpr uint32_t SEQ_Q = 160, SEQ_V = 320, SEQ_GB = 352, SEQ_TOK = 356, SEQ_COL = 20, SEQ_OUT = 32 * SEQ_COL;
constexpr size_t SEQ_SMEM = (2 * GDN_SEQ_CHUNK * (SEQ_TOK + SEQ_OUT) + 2 * SEQ_OUT) * 4;  // tokens, sums of S^T q, sums of S^T k of two tokens
template <bool TILED>
__global__ void __launch_bounds__(256, 1) gdn_seq_k(const __half *cv, const float *la, const float *beta, float *pool, const __half *proj, float *conv,
                                                 __half *oo, const int32_t *sids, gdn_args a, uint32_t HK, uint32_t HV) {
    constexpr int DK = 128, DV = 128, CW = 32, CH = GDN_SEQ_CHUNK;
    extern __shared__ __align__(16) float seq_smem[];
    float *osum = seq_smem + 2 * CH * SEQ_TOK, *msum = osum + 2 * CH * SEQ_OUT;
    pdl_sync();
    const uint32_t cb = blockIdx.x, hv = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = a.nb;
    const uint32_t hk = TILED ? hv % HK : hv / (HV / HK), j = lane & 7, cp = lane >> 3, col = cb * CW + (warp & 3) * 8 + 2 * cp;
    const uint32_t C = 2 * HK * DK + HV * DV;
    const uint32_t slot = (uint32_t)sids[0];
    const bool runs = warp < 4;  // warps 0 .. 3 hold the state: rows 8 j + i and 8 (j + 8) + i of columns col and col + 1
    float *S = pool + (((size_t)slot * a.nlayers + a.layer) * HV + hv) * DK * DV + (size_t)(8 * j) * DV + col;
    const bool pairs = ((uintptr_t)pool & 7) == 0;  // else the two columns one by one: the state is read and written once
    auto get = [&](const float *p) { return pairs ? *(const float2 *)p : make_float2(p[0], p[1]); };
    f32x2 s0[8], s1[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float2 x = runs ? get(S + (size_t)i * DV) : make_float2(0.f, 0.f), y = runs ? get(S + (size_t)(64 + i) * DV) : x;
        s0[i] = pair_of(x.x, y.x);
        s1[i] = pair_of(x.y, y.y);
    }

    // tokens c0 .. of the piece (position tau: row nb - 1 - tau) into their buffer, this warp being number w of `warps`: expressions of gdn_fstep
    auto stage = [&](uint32_t c0, uint32_t w, uint32_t warps) {
        const uint32_t c1 = c0 + CH < nb ? c0 + CH : nb;
        float *buf = seq_smem + (c0 / CH & 1) * CH * SEQ_TOK;
#pragma unroll 4
        for (uint32_t tau = c0 + w; tau < c1; tau += warps) {
            const __half *row = cv + (size_t)(nb - 1 - tau) * C;
            const __half *qh = row + hk * DK, *kh = row + HK * DK + hk * DK;
            const uint2 q4 = *(const uint2 *)(qh + 4 * lane), k4 = *(const uint2 *)(kh + 4 * lane);
            const __half v = row[2 * HK * DK + hv * DV + cb * CW + lane];
            const float lg = la[(size_t)(nb - 1 - tau) * HV + hv], bt = beta[(size_t)(nb - 1 - tau) * HV + hv];
            const float2 qa = __half22float2(*(const __half2 *)&q4.x), qb = __half22float2(*(const __half2 *)&q4.y);
            const float2 ka = __half22float2(*(const __half2 *)&k4.x), kb = __half22float2(*(const __half2 *)&k4.y);
            const float qss = warp_sum(fmaf(qa.x, qa.x, fmaf(qa.y, qa.y, fmaf(qb.x, qb.x, qb.y * qb.y))));
            const float kss = warp_sum(fmaf(ka.x, ka.x, fmaf(ka.y, ka.y, fmaf(kb.x, kb.x, kb.y * kb.y))));
            const float rq_ = rsqrtf(qss / DK + GDN_EPS), rk_ = rsqrtf(kss / DK + GDN_EPS);
            auto qnorm = [&](float x) { return __half2float(__float2half_rn(x * rq_ / DK)); };
            auto knorm = [&](float x) { return __half2float(__float2half_rn(x * rk_ * rsqrtf((float)DK))); };
            // this lane's four rows are rows 4 (lane % 2) .. of row group lane / 2
            float *tk = buf + (tau - c0) * SEQ_TOK, *at = tk + (lane >> 1 & 7) * 20 + 8 * (lane & 1) + (lane >> 4);
            at[0] = knorm(ka.x); at[2] = knorm(ka.y); at[4] = knorm(kb.x); at[6] = knorm(kb.y);
            at += SEQ_Q;
            at[0] = qnorm(qa.x); at[2] = qnorm(qa.y); at[4] = qnorm(qb.x); at[6] = qnorm(qb.y);
            tk[SEQ_V + lane] = __half2float(v);
            if (lane == 0) {
                const float gd = expf(lg);
                *(float4 *)(tk + SEQ_GB) = make_float4(gd, gd, bt, 0.f);
            }
        }
    };
    // 16 group sums in order
    auto sum16 = [](const float *p) {
        float m = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 y = ((const float4 *)p)[i];
            m = i ? m + y.x : y.x;
            m += y.y;
            m += y.z;
            m += y.w;
        }
        return m;
    };
    // outputs whose group sums rounds i0 .. i1 - 1 of the token loop have left, lane = column
    auto outputs = [&](uint32_t i0, uint32_t i1, uint32_t w, uint32_t warps) {
#pragma unroll 4
        for (uint32_t i = i0 + w; i < i1; i += warps) {
            const float o = sum16(osum + (i & (2 * CH - 1)) * SEQ_OUT + lane * SEQ_COL);
            if (i) oo[(size_t)(nb - i) * HV * DV + hv * DV + cb * CW + lane] = __float2half_rn(o);  // (round i: token i - 1)
        }
    };
    stage(0, warp, 8);
    // the conv state after the piece: its last three inputs (channels are spread over the launch's blocks; dn_epi_seq has read the old ones)
    for (uint32_t ch = (hv * 4 + cb) * 256 + tid; ch < C; ch += 4 * HV * 256) {
        float *st = conv + ((size_t)slot * a.nlayers + a.layer) * 3 * C + ch;
        float nw[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int k = (int)nb - 3 + i;  // position in the piece; before it: the old state
            nw[i] = k >= 0 ? __half2float(proj[(size_t)(2 - i) * a.z_stride + ch]) : st[(size_t)(3 + k) * C];
        }
#pragma unroll
        for (int i = 0; i < 3; i++) st[(size_t)i * C] = nw[i];
    }
    __syncthreads();

    auto load8 = [](f32x2 (&x)[8], const float *p) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const ulonglong2 y = ((const ulonglong2 *)p)[i];
            x[2 * i] = y.x;
            x[2 * i + 1] = y.y;
        }
    };
    // the group sums j and j + 8 of this lane's two columns, in the order of the columns of the block
    auto put = [&](float *p, f32x2 m0, f32x2 m1) {
        const float2 x = halves_of(m0), y = halves_of(m1);
        p[j] = x.x;
        p[j + 8] = x.y;
        p[SEQ_COL + j] = y.x;
        p[SEQ_COL + j + 8] = y.y;
    };
    const uint32_t wc = (warp & 3) * 8;  // first column of the warp within the block
    f32x2 qq[8];                         // q of the token before: its S^T q is added up a round later
#pragma unroll
    for (int i = 0; i < 8; i++) qq[i] = 0;
    auto out_sums = [&](uint32_t round) {
        f32x2 o0 = 0, o1 = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            o0 = fma2(s0[i], qq[i], o0);
            o1 = fma2(s1[i], qq[i], o1);
        }
        put(osum + (round & (2 * CH - 1)) * SEQ_OUT + (wc + 2 * cp) * SEQ_COL, o0, o1);
    };
    for (uint32_t c0 = 0; c0 < nb; c0 += CH) {
        const uint32_t c1 = c0 + CH < nb ? c0 + CH : nb;
        if (!runs) {
            if (c1 < nb) stage(c1, warp - 4, 4);
            if (c0) outputs(c0 - CH, c0, warp - 4, 4);
        } else {
            const float *tk = seq_smem + (c0 / CH & 1) * CH * SEQ_TOK;
            f32x2 kk[8];
            load8(kk, tk + 20 * j);
            float4 gb = *(const float4 *)(tk + SEQ_GB);
            float v = tk[SEQ_V + wc + j];
#pragma unroll 2
            for (uint32_t tau = c0; tau < c1; tau++) {
                f32x2 d0[8], d1[8], m0 = 0, m1 = 0;
                const f32x2 gg = pair_of(gb.x, gb.y);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    d0[i] = mul2(s0[i], gg);
                    d1[i] = mul2(s1[i], gg);
                    m0 = fma2(d0[i], kk[i], m0);
                    m1 = fma2(d1[i], kk[i], m1);
                }
                float *ms = msum + (tau & 1) * SEQ_OUT + wc * SEQ_COL;  // two of them: a warp barrier lies between a read and the next write
                put(ms + 2 * cp * SEQ_COL, m0, m1);
                __syncwarp();
                const float mt = sum16(ms + j * SEQ_COL);  // lanes j, j + 8, ..: column j of the warp
                out_sums(tau);                             // (of the token before)
                const float *tn = tau + 1 < c1 ? tk + SEQ_TOK : tk;
                load8(qq, tk + SEQ_Q + 20 * j);
                const float d = gb.z * (v - mt);
                const float da = __shfl_sync(0xffffffffu, d, 2 * cp), db = __shfl_sync(0xffffffffu, d, 2 * cp + 1);
                const f32x2 dd0 = pair_of(da, da), dd1 = pair_of(db, db);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    s0[i] = fma2(kk[i], dd0, d0[i]);
                    s1[i] = fma2(kk[i], dd1, d1[i]);
                }
                tk = tn;  // the next token's operands (the last one reads its own again)
                load8(kk, tk + 20 * j);
                gb = *(const float4 *)(tk + SEQ_GB);
                v = tk[SEQ_V + wc + j];
            }
        }
        __syncthreads();
    }
    auto put_state = [&](float *p, float a0, float a1) {
        if (pairs) *(float2 *)p = make_float2(a0, a1);
        else {
            p[0] = a0;
            p[1] = a1;
        }
    };
    if (runs) {
        out_sums(nb);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float2 x = halves_of(s0[i]), y = halves_of(s1[i]);
            put_state(S + (size_t)i * DV, x.x, y.x);
            put_state(S + (size_t)(64 + i) * DV, x.y, y.y);
        }
    }
    __syncthreads();
    outputs((nb - 1) / CH * CH, nb + 1, warp, 8);
}

static cudaError_t launch_gdn_seq(const QwLaunch &L) {
    const uint32_t HK = (uint32_t)L.def("HK", 16), HV = (uint32_t)L.def("HV", 32), DK = (uint32_t)L.def("DK", 128), DV = (uint32_t)L.def("DV", 128);
    const bool tiled = L.def("GDN_TILED", 1) != 0;
    const uint32_t C = 2 * HK * DK + HV * DV;
    gdn_args a = L.bytes<gdn_args>(8);
    QW_CHECK_ARG(DK == 128 && DV == 128 && HV % HK == 0 && L.has_bytes(8, 16) && a.nb >= 1 && a.nb <= GDN_SEQ_MAX && a.layer < a.nlayers && a.z_stride >= C);
    for (int i = 0; i <= 7; i++) QW_CHECK_ARG(L.buf<void>(i) != nullptr);
    QW_CHECK_ARG(L.avail(0) >= (size_t)a.nb * C * 2 && L.avail(1) >= (size_t)a.nb * HV * 4 && L.avail(2) >= (size_t)a.nb * HV * 4 &&
                 L.avail(4) >= ((size_t)(a.nb - 1) * a.z_stride + C) * 2 && L.avail(6) >= (size_t)a.nb * HV * DV * 2 && L.avail(7) >= 4);
    auto kern = tiled ? gdn_seq_k<true> : gdn_seq_k<false>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEQ_SMEM);
    if (e != cudaSuccess) return e;
    qw_launch(kern, dim3(4, HV), 256, SEQ_SMEM, L.stream, L.buf<__half>(0), L.buf<float>(1), L.buf<float>(2), L.buf<float>(3), L.buf<__half>(4), L.buf<float>(5),
              L.buf<__half>(6), L.buf<int32_t>(7), a, HK, HV);
    return cudaGetLastError();
}
QW_FAMILY(gdn_seq, launch_gdn_seq, 256)

// Gated RMSNorm of gdn_seq's output, in the expressions of gdn_fstep: y = o * rsqrt(mean o^2 + eps) * w * sigmoid(z), in place.
// A warp takes a head of a token, four columns per lane 32 apart; its four sums of 32 squares are the four warps' of gdn_fstep.  (A block of four warps per head and token
// met once in shared memory for 128 values: 419 tokens 15.9 -> 6.3 us on a B200.)
// binds: 0 = o fp16 [nb][HV*DV] (becomes y), 4 = z fp16 (row stride z_stride), 5 = norm weight fp32 [DV], 8 = gdn_args.  grid ceil(HV nb / 4) x 128
__global__ void __launch_bounds__(128) gdn_gate_k(__half *o, const __half *z, const float *nw, gdn_args a, uint32_t HV) {
    constexpr int DV = 128;
    pdl_launch();
    const uint32_t lane = threadIdx.x & 31, n = blockIdx.x * 4 + (threadIdx.x >> 5);
    float wv[4];
#pragma unroll
    for (int i = 0; i < 4; i++) wv[i] = nw[32 * i + lane];
    pdl_wait();
    if (n >= a.nb * HV) return;
    const uint32_t t = n / HV, hv = n % HV;
    __half *p = o + (size_t)n * DV + lane;
    const __half *zp = z + (size_t)t * a.z_stride + hv * DV + lane;
    float x[4], zz[4], ss[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        zz[i] = __half2float(zp[32 * i]);
        x[i] = __half2float(p[32 * i]);
        ss[i] = x[i] * x[i];
    }
#pragma unroll
    for (int off = 16; off; off >>= 1)
#pragma unroll
        for (int i = 0; i < 4; i++) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], off);
    const float r = rsqrtf((((ss[0] + ss[1]) + ss[2]) + ss[3]) / DV + GDN_EPS);
#pragma unroll
    for (int i = 0; i < 4; i++) p[32 * i] = __float2half_rn(x[i] * r * wv[i] * (1.0f / (1.0f + expf(-zz[i]))));
}
// Up to 64 rows: a block of four warps per head and token (prompts of 45 tokens, 12 layers: 2.42 ms, with the other form 2.47)
__global__ void __launch_bounds__(128) gdn_gate_few_k(__half *o, const __half *z, const float *nw, gdn_args a, uint32_t HV) {
    constexpr int DV = 128;
    __shared__ float red[4];
    pdl_sync();
    const uint32_t hv = blockIdx.x, t = blockIdx.y, c = threadIdx.x, lane = c & 31, warp = c >> 5;
    __half *p = o + (size_t)t * HV * DV + hv * DV + c;
    const float zz = __half2float(z[(size_t)t * a.z_stride + hv * DV + c]);
    const float x = __half2float(*p);
    const float ss = warp_sum(x * x);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    const float r = rsqrtf((((red[0] + red[1]) + red[2]) + red[3]) / DV + GDN_EPS);
    *p = __float2half_rn(x * r * nw[c] * (1.0f / (1.0f + expf(-zz))));
}
static cudaError_t launch_gdn_gate(const QwLaunch &L) {
    const uint32_t HV = (uint32_t)L.def("HV", 32), DV = (uint32_t)L.def("DV", 128);
    gdn_args a = L.bytes<gdn_args>(8);
    QW_CHECK_ARG(DV == 128 && L.has_bytes(8, 16) && a.nb >= 1 && a.nb <= GDN_SEQ_MAX && a.z_stride >= HV * DV);
    QW_CHECK_ARG(L.buf<void>(0) && L.buf<void>(4) && L.buf<void>(5) && L.avail(0) >= (size_t)a.nb * HV * DV * 2 &&
                 L.avail(4) >= ((size_t)(a.nb - 1) * a.z_stride + HV * DV) * 2 && L.avail(5) >= DV * 4);
    if (a.nb <= 64) qw_launch(gdn_gate_few_k, dim3(HV, a.nb), 128, 0, L.stream, L.buf<__half>(0), L.buf<__half>(4), L.buf<float>(5), a, HV);
    else qw_launch(gdn_gate_k, (a.nb * HV + 3) / 4, 128, 0, L.stream, L.buf<__half>(0), L.buf<__half>(4), L.buf<float>(5), a, HV);
    return cudaGetLastError();
}
QW_FAMILY(gdn_gate, launch_gdn_gate, 128)
