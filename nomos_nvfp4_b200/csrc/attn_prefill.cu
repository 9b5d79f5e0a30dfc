// Host side of the query-major prefill kernel (attn_prefill_kernel.cuh): instance choice and launch.  Which calls come
// here is decided in attn_fused.cu (prefill_eligible).
#include <cstring>

#include "attn_prefill_kernel.cuh"

namespace nomos {

using fused::LOG2E;

namespace {

template <int HD, int FMT, int QL, int NQ>
static int launch_prefill_inst(cudaStream_t st, const AttnArgs &a, unsigned int *fault) {
    using C = pf::Cfg<HD, FMT, QL, NQ>;
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_set[dev]) {
        cudaFuncSetAttribute(pf::attn_prefill_kernel<HD, FMT, QL, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        attr_set[dev] = true;
    }
    pf::PParams p;
    std::memset(&p, 0, sizeof(p));
    p.q = static_cast<const uint8_t *>(a.q);
    p.out = static_cast<uint8_t *>(a.out);
    p.k_cache = static_cast<const uint8_t *>(a.k_cache);
    p.v_cache = static_cast<const uint8_t *>(a.v_cache);
    p.k_scales = static_cast<const uint8_t *>(a.k_scales);
    p.v_scales = static_cast<const uint8_t *>(a.v_scales);
    p.out_type = a.out_type;
    p.batch = a.batch; p.S = a.S; p.nh = a.nh; p.nkv = a.nkv; p.kvg = a.kvg; p.cache_cap = a.cache_cap;
    p.row_bytes = FMT == KV_I8 ? a.cache_hd : a.cache_hd / 2;
    p.row0 = a.win_start % a.cache_cap;
    p.key_len = a.klen;
    p.d0 = a.d0_set ? a.d0 : a.klen - a.S;
    p.window = a.window;
    p.pos_per_tile = pf::MR / a.kvg;
    p.q_blocks = (a.S + C::NQ * p.pos_per_tile - 1) / (C::NQ * p.pos_per_tile);
    p.q_scale = a.softmax_scale * LOG2E;
    p.q_batch_stride = a.q_batch_stride; p.out_batch_stride = a.out_batch_stride;
    p.kv_batch_stride = a.kv_batch_stride; p.scale_batch_stride = a.scale_batch_stride;
    p.fault = fault;
    if (p.fault == nullptr) { set_error("attn_prefill: device fault word unavailable"); return NOMOS_ECUDA; }
    const long ctas = (long)p.q_blocks * a.nkv * C::DSPLIT * a.batch;
    if (ctas >= (1l << 31)) { set_error("attn_prefill: too many query blocks"); return NOMOS_EUNSUPPORTED; }
    cudaLaunchAttribute pdl[1];
    pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(C::NTHREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = st;
    cfg.attrs = pdl; cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, pf::attn_prefill_kernel<HD, FMT, QL, NQ>, p);
    if (e != cudaSuccess) { set_error("attn_prefill launch: %s", cudaGetErrorString(e)); return NOMOS_ECUDA; }
    return NOMOS_OK;
}

template <int FMT>
static int launch_prefill_fmt(cudaStream_t st, const AttnArgs &a, int query_tiles, unsigned int *fault) {
    const bool one = a.q_type == ET_BF16;              // bf16 query rows fit one fp16 limb exactly
    switch (a.l_hd) {
        case 128:
            if (query_tiles == 1) return one ? launch_prefill_inst<128, FMT, 1, 1>(st, a, fault) : launch_prefill_inst<128, FMT, 2, 1>(st, a, fault);
            return one ? launch_prefill_inst<128, FMT, 1, 2>(st, a, fault) : launch_prefill_inst<128, FMT, 2, 2>(st, a, fault);
        case 256: return one ? launch_prefill_inst<256, FMT, 1, 1>(st, a, fault) : launch_prefill_inst<256, FMT, 2, 1>(st, a, fault);
        default: return launch_prefill_inst<512, FMT, 1, 1>(st, a, fault);
    }
}

}  // namespace

int launch_attn_prefill(cudaStream_t st, const AttnArgs &a, int query_tiles, unsigned int *fault) {
    switch (a.kv_fmt) {
        case KV_I8: return launch_prefill_fmt<KV_I8>(st, a, query_tiles, fault);
        case KV_I4: return launch_prefill_fmt<KV_I4>(st, a, query_tiles, fault);
        default: return launch_prefill_fmt<KV_I4B32>(st, a, query_tiles, fault);
    }
}

}  // namespace nomos
