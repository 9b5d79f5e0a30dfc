// Attention over an UNQUANTISED (fp32 or bf16) KV cache: single-token GQA decode
// and the prefix-batched (verify / chunked-prefill) form, sm_100a.
//
// These are the legacy KV modes of the reference (two cuBLAS strided-batched GEMMs
// with a softmax kernel between them, scores materialised in HBM):
//   lib/attention_gpu.mojo:165-204 (fp32), :207-248 (bf16 operands)
//   lib/batched_attn_gpu.mojo:499-548 (fp32 prefix), :613-666 (bf16 prefix)
//   masks: lib/batched_attn_gpu.mojo:285-409
// Here they are one split-K streaming kernel and a merge of the splits: a row of K or V is 16 or 32 lanes of 16-byte loads, a
// warp has four (two for the widest rows) such row groups of K and of V in flight, keeps the GQA group's query rows in
// registers and carries (m, l, o) online; nothing is written to HBM but the partials.  Arithmetic is fp32 on the stored
// values (bf16 widens exactly).
#include <math_constants.h>

#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace nomos {
namespace {

constexpr int DW = 4;                 // warps per CTA
constexpr float LOG2E = 1.4426950408889634f;
constexpr float M_INIT = -1.0e30f;

struct DParams {
    const float *q;
    const uint8_t *k, *v;
    float *out;
    float *part_o, *part_ml;          // split partials: [splits][rows][HD], then [splits][rows] (m in log2 units, l)
    int S, nh, nkv, kvg, cache_hd, max_seq, key_len, window, query_base_pos, key_base_pos;
    int splits, keys_per_split, grows;
};

template <typename T>
__device__ __forceinline__ void widen(const uint4 &w, float (&x)[16 / sizeof(T)]) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (sizeof(T) == 4) {
            x[i] = __uint_as_float(u[i]);
        } else {
            x[2 * i] = __uint_as_float(u[i] << 16);
            x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
    }
}

// grid = (splits, nkv * subgroups, S); one CTA = one KV head, one query row and KVG of
// the group's query heads (a GQA group wider than KVG is covered by several CTAs).
// Memory-bound: with one key row per warp and step (the loads of the next key issued after this key's reductions) a bf16
// cache of 8192 keys x 16 heads x 128 (67 MB) took 54 us; with eight rows of K and of V in flight per warp and the merge
// chained behind it 19.4 us.  256 rows behind 1792 keys: 839 -> 480 us (fp32 FMA and L2 traffic: a CTA per query row).
template <typename T, int HD, int KVG>
__global__ void __launch_bounds__(DW * 32) attn_dense_kernel(const DParams p) {
    constexpr int EPL = 16 / (int)sizeof(T);                           // elements per 16-byte load
    constexpr int LPR = HD / EPL < 32 ? HD / EPL : 32;                 // lanes per row
    constexpr int NC = HD / (EPL * LPR);                               // loads per lane and row
    constexpr int KPW = 32 / LPR;                                      // keys side by side in a warp
    constexpr int U = NC >= 4 ? 2 : 4;                                 // key steps in flight
    constexpr int NST = DW * KPW;                                      // (m, l, o) states per CTA
    __shared__ float so[NST][KVG][HD];
    __shared__ float sml[NST][KVG][2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / LPR, ln = lane % LPR;
    const int nsub = p.kvg / KVG;
    const int split = blockIdx.x, kvh = blockIdx.y / nsub, s = blockIdx.z;
    const int h0 = kvh * p.kvg + (blockIdx.y % nsub) * KVG;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

    // valid key range of row s (lib/batched_attn_gpu.mojo:314-326)
    const int q_abs = p.query_base_pos + s;
    const int hi = min(q_abs - p.key_base_pos, p.key_len - 1);
    int lo = (p.window > 0 && q_abs - p.window + 1 > 0) ? q_abs - p.window + 1 : 0;
    lo = max(lo - p.key_base_pos, 0);
    const int k_begin = max(lo, split * p.keys_per_split);
    const int k_end = min(hi + 1, (split + 1) * p.keys_per_split);

    float q[KVG][NC][EPL], acc[KVG][NC][EPL], M[KVG], l[KVG];
#pragma unroll
    for (int j = 0; j < KVG; ++j) {
        M[j] = M_INIT; l[j] = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int i = 0; i < EPL; ++i) {
                q[j][c][i] = p.q[((size_t)s * p.nh + h0 + j) * HD + (c * LPR + ln) * EPL + i] * LOG2E;
                acc[j][c][i] = 0.0f;
            }
    }
    const uint8_t *kb = p.k + ((size_t)kvh * p.max_seq * p.cache_hd + ln * EPL) * sizeof(T);
    const uint8_t *vb = p.v + ((size_t)kvh * p.max_seq * p.cache_hd + ln * EPL) * sizeof(T);
    const size_t pitch = (size_t)p.cache_hd * sizeof(T);
    for (int key0 = k_begin + warp * (KPW * U); key0 < k_end; key0 += DW * KPW * U) {
        uint4 kx[U][NC], vx[U][NC];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t off = (size_t)min(key0 + u * KPW + sub, k_end - 1) * pitch;
#pragma unroll
            for (int c = 0; c < NC; ++c) kx[u][c] = *reinterpret_cast<const uint4 *>(kb + off + c * LPR * 16);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int key = key0 + u * KPW + sub;                      // (no value row beyond the split: zero weight x infinity is not zero)
#pragma unroll
            for (int c = 0; c < NC; ++c)
                vx[u][c] = key < k_end ? *reinterpret_cast<const uint4 *>(vb + (size_t)key * pitch + c * LPR * 16) : make_uint4(0u, 0u, 0u, 0u);
        }
        float sc[U][KVG];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int j = 0; j < KVG; ++j) sc[u][j] = 0.0f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float x[EPL];
                widen<T>(kx[u][c], x);
#pragma unroll
                for (int j = 0; j < KVG; ++j)
#pragma unroll
                    for (int i = 0; i < EPL; ++i) sc[u][j] = fmaf(q[j][c][i], x[i], sc[u][j]);
            }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < KVG; ++j) sc[u][j] += __shfl_xor_sync(0xffffffffu, sc[u][j], o);
        float pe[U][KVG], alpha[KVG];
#pragma unroll
        for (int j = 0; j < KVG; ++j) {
            float m_new = M[j];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (key0 + u * KPW + sub >= k_end) sc[u][j] = -CUDART_INF_F;
                m_new = fmaxf(m_new, sc[u][j]);
            }
            alpha[j] = ex2f(M[j] - m_new);
            l[j] *= alpha[j];
#pragma unroll
            for (int u = 0; u < U; ++u) { pe[u][j] = ex2f(sc[u][j] - m_new); l[j] += pe[u][j]; }
            M[j] = m_new;
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
#pragma unroll
            for (int j = 0; j < KVG; ++j)
#pragma unroll
                for (int i = 0; i < EPL; ++i) acc[j][c][i] *= alpha[j];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float x[EPL];
                widen<T>(vx[u][c], x);
#pragma unroll
                for (int j = 0; j < KVG; ++j)
#pragma unroll
                    for (int i = 0; i < EPL; ++i) acc[j][c][i] = fmaf(pe[u][j], x[i], acc[j][c][i]);
            }
        }
    }

    const int st = warp * KPW + sub;
#pragma unroll
    for (int j = 0; j < KVG; ++j) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int i = 0; i < EPL; ++i) so[st][j][(c * LPR + ln) * EPL + i] = acc[j][c][i];
        if (ln == 0) { sml[st][j][0] = M[j]; sml[st][j][1] = l[j]; }
    }
    __syncthreads();
#pragma unroll 1
    for (int j = 0; j < KVG; ++j) {
        float mstar = M_INIT;
#pragma unroll
        for (int w = 0; w < NST; ++w) mstar = fmaxf(mstar, sml[w][j][0]);
        float wgt[NST], lstar = 0.0f;
#pragma unroll
        for (int w = 0; w < NST; ++w) { wgt[w] = ex2f(sml[w][j][0] - mstar); lstar += wgt[w] * sml[w][j][1]; }
        const long grow = (long)s * p.nh + h0 + j;
        for (int d = threadIdx.x; d < HD; d += DW * 32) {
            float o = 0.0f;
#pragma unroll
            for (int w = 0; w < NST; ++w) o += wgt[w] * so[w][j][d];
            if (p.splits > 1) p.part_o[((size_t)split * p.grows + grow) * HD + d] = o;
            else p.out[grow * HD + d] = lstar == 0.0f ? 0.0f : o / lstar;      // (a NaN stays one)
        }
        if (p.splits > 1 && threadIdx.x == 0) {
            p.part_ml[((size_t)split * p.grows + grow) * 2] = mstar;
            p.part_ml[((size_t)split * p.grows + grow) * 2 + 1] = lstar;
        }
    }
}

// Merge of the splits: one CTA per query row, NG groups of threads over the splits.
constexpr int MERGE_MAX = 512;        // most splits
template <int HD>
__global__ void __launch_bounds__(256) dense_merge_kernel(const DParams p) {
    constexpr int LPR = HD / 4 < 64 ? HD / 4 : 64, NG = 256 / LPR, NC = HD / (4 * LPR);
    __shared__ float wgt[MERGE_MAX];
    __shared__ float red[16];
    __shared__ float4 part[NG][HD / 4];
    const int tid = threadIdx.x, row = blockIdx.x, warp = tid >> 5;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    float m = M_INIT;
    for (int i = tid; i < p.splits; i += 256) m = fmaxf(m, p.part_ml[((size_t)i * p.grows + row) * 2]);
    m = warp_max(m);
    if ((tid & 31) == 0) red[warp] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) m = fmaxf(m, red[w]);
    float l = 0.0f;
    for (int i = tid; i < p.splits; i += 256) {
        const float2 ml = *reinterpret_cast<const float2 *>(p.part_ml + ((size_t)i * p.grows + row) * 2);
        const float w = ml.y == 0.0f ? 0.0f : ex2f(ml.x - m);          // (no key in the split; a NaN stays one)
        wgt[i] = w;
        l = fmaf(w, ml.y, l);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((tid & 31) == 0) red[8 + warp] = l;
    __syncthreads();
    l = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) l += red[8 + w];
    const int g = tid / LPR, ln = tid % LPR;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
        for (int i = g; i < p.splits; i += NG) {
            const float4 x = *reinterpret_cast<const float4 *>(p.part_o + ((size_t)i * p.grows + row) * HD + 4 * (c * LPR + ln));
            const float w = wgt[i];
            if (w != 0.0f) { o.x = fmaf(w, x.x, o.x); o.y = fmaf(w, x.y, o.y); o.z = fmaf(w, x.z, o.z); o.w = fmaf(w, x.w, o.w); }
        }
        part[g][c * LPR + ln] = o;
    }
    __syncthreads();
    for (int d = tid; d < HD; d += 256) {
        float o = 0.0f;
#pragma unroll
        for (int k = 0; k < NG; ++k) o += reinterpret_cast<const float *>(part[k])[d];
        p.out[(size_t)row * HD + d] = l == 0.0f ? 0.0f : o / l;
    }
}

template <typename T, int HD, int KVG>
static int launch_dense_inst(cudaStream_t st, const DenseAttnArgs &a) {
    static int occ[64] = {0}, sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (occ[dev] == 0) {
        int n = 0, sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, attn_dense_kernel<T, HD, KVG>, DW * 32, 0);
        cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
        sms[dev] = sm > 0 ? sm : 148;
        occ[dev] = n > 0 ? n : 1;
    }
    const int grows = a.S * a.nh;
    const long units = (long)a.nkv * (a.kvg / KVG) * a.S;
    // one resident wave of CTAs, each with at least two rounds of its warps' loads
    int splits = (int)std::max<long>(1, (long)sms[dev] * std::min(occ[dev], 8) / std::max<long>(1, units));
    splits = std::min({splits, std::max(1, a.key_len / (DW * 16)), MERGE_MAX});
    // partials live in the caller's scratch, which is sized for the reference's scores: fewer splits when it is small
    const uintptr_t ws0 = (reinterpret_cast<uintptr_t>(a.workspace) + 15) & ~(uintptr_t)15;
    const long ws_bytes = a.workspace ? a.ws_bytes - (long)(ws0 - reinterpret_cast<uintptr_t>(a.workspace)) : 0;
    const long per_split = (long)grows * (HD + 2) * 4;
    if (splits > 1 && per_split * splits > ws_bytes) splits = (int)std::max<long>(1, ws_bytes / per_split);
    const int kps = (a.key_len + splits - 1) / splits;
    splits = (a.key_len + kps - 1) / kps;
    DParams p;
    p.q = a.q; p.k = static_cast<const uint8_t *>(a.k_cache); p.v = static_cast<const uint8_t *>(a.v_cache);
    p.out = a.out; p.part_o = reinterpret_cast<float *>(ws0); p.part_ml = p.part_o + (size_t)splits * grows * HD;
    p.S = a.S; p.nh = a.nh; p.nkv = a.nkv; p.kvg = a.kvg; p.cache_hd = a.cache_hd; p.max_seq = a.max_seq;
    p.key_len = a.key_len; p.window = a.window; p.query_base_pos = a.query_base_pos; p.key_base_pos = a.key_base_pos;
    p.splits = splits; p.keys_per_split = kps; p.grows = grows;
    cudaLaunchAttribute pdl[1];
    pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, a.nkv * (a.kvg / KVG), a.S); cfg.blockDim = dim3(DW * 32); cfg.stream = st;
    cfg.attrs = pdl; cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, attn_dense_kernel<T, HD, KVG>, p);
    if (e == cudaSuccess && splits > 1) {
        cfg.gridDim = dim3(grows); cfg.blockDim = dim3(256);
        e = cudaLaunchKernelEx(&cfg, dense_merge_kernel<HD>, p);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("attn_dense launch: %s", cudaGetErrorString(e)); return NOMOS_ECUDA; }
    return NOMOS_OK;
}

template <typename T>
static int dispatch_dense(cudaStream_t st, const DenseAttnArgs &a) {
    // heads of one GQA group handled per CTA: 4 / 2 / 1, whichever divides kvg
#define NOMOS_DENSE(HD_)                                                              \
    if (a.l_hd == HD_) {                                                              \
        if (HD_ <= 256 && a.kvg % 4 == 0) return launch_dense_inst<T, HD_, 4>(st, a); \
        if (a.kvg % 2 == 0) return launch_dense_inst<T, HD_, 2>(st, a);               \
        return launch_dense_inst<T, HD_, 1>(st, a);                                   \
    }
    NOMOS_DENSE(128) NOMOS_DENSE(256) NOMOS_DENSE(512)
#undef NOMOS_DENSE
    set_error("dense attention: head_dim %d unsupported (128, 256, 512)", a.l_hd);
    return NOMOS_EUNSUPPORTED;
}

}  // namespace

int launch_attn_dense(cudaStream_t st, const DenseAttnArgs &a) {
    return a.kv_is_bf16 ? dispatch_dense<__nv_bfloat16>(st, a) : dispatch_dense<float>(st, a);
}

}  // namespace nomos
