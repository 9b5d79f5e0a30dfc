// Query-major flash prefill straight off the packed KV cache on the fifth-generation tensor cores (tcgen05 + tensor
// memory), sm_100a: int8, int4 and block-32 int4 caches, head dims 128 / 256 / 512.  Which calls come here
// is decided in attn_fused.cu, the launch is in attn_prefill.cu.
//
// Replaces the reference's square / prefix batched prefill attention
//   lib/attention_gpu_int8.mojo:804-887 (int8), lib/batched_attn_gpu.mojo:448-666 (fp32 / bf16 twins)
// which materialise an [nkv, S*kvg, key_len] score matrix in device memory (the reference's own note on the
// "real fix": lib/engine_prefill.mojo:145; the cap it forces on prompts: pyhost/serve.py:41-64).  Nothing of size
// S x key_len exists here: a CTA owns 128 or 256 query rows and walks the key tiles they may attend.
//
// A query tile = 128 rows of ONE KV head: 128 / kvg consecutive query positions x the kvg query heads of the group
// (position-major, so causal bounds are monotone in the row index).  Per key tile of KT keys:
//   S[128 x KT]  = Q16[128 x HD] (A, shared memory) x K16[KT x HD]^T (B, K-major)           kind::f16, fp32 accumulate
//   O[128 x DV] += P16[128 x KT] (A, TENSOR memory) x V16[KT x DV] (B, MN-major: [key][dim] as stored)
// Operands are fp16 and carry all the bits of what they stand for:
//   Q16  the query row times a power of two of its own (bf16 rows fit one fp16 exactly; fp32 rows take hi + lo, 22 bits)
//   K16, V16  the cache CODES (exact in fp16), row scales applied in fp32 afterwards; block-32 rows: code x fp16 block
//        scale is up to 14 bits, split into code x (top 7 bits of the scale) + code x (the other 4), both exact
//   P16  the softmax weight times the value's row scale as hi + lo (22 bits)
// The value scale rides in the exponent: with u' = logit + log2(vscale) the weight is w = 2^(u' - m), m a whole-number
// running reference of u', so w fits fp16 whatever the scale, and the denominator takes w / vscale.
//
// Roles: per query tile eight softmax warps of 16 rows (a thread holds two rows and every fourth pair of keys; the weights
// go back into the SAME columns as S, hi and lo, as the A operand of PV); "dequant" warps in teams of two that fetch cache
// bytes from global memory ahead of their turn, widen them and fill a ring of K / V slots in the order the tensor core
// takes them (rows are addressed one by one: rings may wrap); one MMA warp.  head_dim 128: one query tile per CTA, or two
// in turn, one tile's softmax under the other's products; at 512 two CTAs per query tile that each own 256 output dims.
// Four S buffers, shared by the query tiles; the order of products and waits is prefill_schedule.h.  O stays in tensor
// memory; it is rescaled in place only when a row's reference moves, which happens when a chunk exceeds it by more than
// 2^8 (a handful of times per row).
// Every wait is an mbarrier wait with a time limit; a wait that runs out raises the CTA's abort flag and bit 1 of the
// device fault word, every role leaves its loop, tensor memory is freed and the CTA exits.
#pragma once

#include "attn_tc5_kernel.cuh"
#include "prefill_schedule.h"

namespace nomos {
namespace pf {

using fused::LOG2E;
using tc5::wait_or_abort;

constexpr int MR = 128;                       // query rows per tile = M of the MMAs
constexpr float M_INIT = -1.0e30f;
constexpr float LAZY = 8.0f;                  // base-2 slack before a row's running reference is moved
constexpr float VS_MIN = 1.0e-30f;            // value scales of smaller size count as this (1 / scale stays finite)
constexpr int KT = 64;                        // keys per tile
constexpr int SMEM_MAX = 232448;              // shared memory a CTA may ask for

constexpr int cmin(int a, int b) { return a < b ? a : b; }

template <int HD_, int FMT_, int QL_, int NQ_>
struct Cfg {
    static constexpr int HD = HD_, FMT = FMT_, QL = QL_;               // QL: fp16 limbs of the query
    static constexpr int KL = FMT == KV_I4B32 ? 2 : 1;                 // fp16 limbs of K and V
    // Query tiles per CTA.  Two share a CTA's K and V slots at head_dim 128 (64 keys x 256 rows 1.45 us, 128 rows 1.05 us), but
    // where all query tiles find an SM of their own the CTA with one is done sooner.
    static constexpr int NQ = NQ_;
    static_assert(NQ == 1 || (NQ == 2 && HD == 128), "tensor memory columns");
    static constexpr int DV = cmin(HD, 256);                           // output dims per CTA
    static constexpr int DSPLIT = HD / DV;
    static constexpr int Q_BLOCK = MR * 128;                           // 64 dims of a query tile (one swizzle block column)
    static constexpr int Q_LIMB = Q_BLOCK * (HD / 64);
    static constexpr int Q_BYTES = NQ * QL * Q_LIMB;
    static_assert(Q_BYTES <= 131072, "the query tiles stay resident");
    static constexpr int BLOCK = KT * 128;                             // 64 dims of KT keys
    static constexpr int SLOT = 2 * BLOCK;                             // ring slot: KT keys x 128 dims, fp16
    static constexpr int KS = HD / 128 * KL, VS = DV / 128 * KL;       // slots of a K tile, of a V tile
    // Per-key constants of tile i are overwritten at tile i + nconst, behind the wait for that tile's first K slot, which
    // the ring grants only once V of tile i is released (all softmax rows of tile i are then done): ring order
    // K0 K1 V0 K2 V1 ... makes that (nconst - 2) * (KS + VS) >= slots - 1.
    static constexpr int nconst(int slots) { return 2 + (slots - 1 + KS + VS - 1) / (KS + VS); }
    static constexpr int CONST_BYTES = 3 * KT * 4 + 8;                 // per-key constants of a tile, and a bit per key
    static constexpr int smem(int slots) { return Q_BYTES + slots * SLOT + nconst(slots) * CONST_BYTES + (2 * slots + nconst(slots) + 3 * 4 + 1) * 8 + 16; }
    static constexpr int most_slots() { int n = 2 * KL; while (smem(n + KL) <= SMEM_MAX) n += KL; return n; }
    static constexpr int NSLOT = most_slots(), NCONST = nconst(NSLOT);
    static_assert(NSLOT >= 2 * KL && NSLOT % KL == 0, "a V unit and the K unit behind it; the limbs of a unit side by side");
    static constexpr int NB = s_buffers<NQ>(), NSB = NB * NQ;          // S buffers per query tile, in all
    static constexpr int TMEM_O = 0, TMEM_S = 256;
    static_assert(NQ * DV <= 256 && NSB * KT <= 256, "tensor memory columns");
    static constexpr int NSW = 8 * NQ;                                 // softmax warps: two per 32 TMEM lanes, 16 rows each
    // Dequant warps, in teams of two that take the units (KL slots) in turn: what a unit costs a team besides its bytes
    // (slot wait, address arithmetic, proxy fence, hand-off: about 1500 cycles) overlaps the other teams'.
    // No more teams than the ring holds units: a slot's next user may not wait for a phase of its barrier whose
    // predecessor is still pending (products release the slots in order, so with this many none can).
    static constexpr int TEAMS = cmin(NQ == 2 ? 3 : 5, NSLOT / KL), ND = 2 * TEAMS;
    static constexpr int W_DEQ = NSW, W_MMA = NSW + ND;
    static constexpr int NTHREADS = 32 * (NSW + ND + 1);
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_RING = Q_BYTES;
    // [NCONST]: fp32 [KT] each of logit factor, log2(vs) and 1 / vs, vs = |value scale|; then the keys with a negative one
    static constexpr int OFF_CONST = OFF_RING + NSLOT * SLOT;
    static constexpr int OFF_BAR = OFF_CONST + NCONST * CONST_BYTES;
    static constexpr int NBAR = 2 * NSLOT + NCONST + 3 * NSB + 1;
    static constexpr int OFF_MISC = OFF_BAR + NBAR * 8;
    static constexpr int SMEM_BYTES = OFF_MISC + 16;                   // (no static shared memory: the dynamic part starts 1024-byte aligned)
    static_assert(SMEM_BYTES == smem(NSLOT) && SMEM_BYTES <= SMEM_MAX, "shared memory budget of a CTA");
    // dequant work of a slot: 16-byte pieces of cache bytes
    static constexpr int CPP = FMT == KV_I8 ? 16 : 32;                 // codes per piece
    static constexpr int PPR = 128 / CPP;                              // pieces per row of a slot
    static constexpr int NP = KT * PPR / 64;                           // pieces per thread and slot
    static constexpr int NBW = HD / 64;                                // block-32: 32-bit words of fp16 scales per row
};

struct PParams {
    const uint8_t *q;
    uint8_t *out;
    const uint8_t *k_cache, *v_cache, *k_scales, *v_scales;
    int out_type;
    int batch, S, nh, nkv, kvg, cache_cap;
    int row_bytes;                            // bytes of a cache row
    int row0;                                 // ring slot of key index 0 of the array
    int key_len;                              // keys of the array
    int d0;                                   // query row s may attend key indices <= d0 + s (d0 may be negative)
    int window;                               // > 0: and no key index below d0 + s - window + 1
    int pos_per_tile;                         // 128 / kvg
    int q_blocks;
    float q_scale;                            // softmax_scale * log2(e)
    long q_batch_stride, out_batch_stride, kv_batch_stride, scale_batch_stride;
    unsigned int *fault;
};

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// A operand in tensor memory (fp16 pairs in 32-bit columns, lane = row)
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Instruction descriptor for kind::f16: fp32 accumulate, fp16 A and B, M = 128, given N; B may be MN-major.
__device__ __forceinline__ constexpr uint32_t make_idesc_f16(int n, bool b_mn_major) {
    return (1u << 4) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(pred));
    return pred != 0;
}
// 16 lanes x 8 n columns, spread over the warp like an MMA accumulator: registers 4 e + 2 r + {0, 1} of a thread are
// columns 8 e + 2 (lane % 4) + {0, 1} of row 8 r + lane / 4.  The caller waits.
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_frag32(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// The same rows, packed pairs: register 2 e + r is column 4 e + lane % 4 of row 8 r + lane / 4.
__device__ __forceinline__ void tmem_st_pairs32(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// two floats per instruction
struct __align__(8) F2 { float x, y; };
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 d;
    asm("{\n.reg .b64 ra, rb, rc, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nmov.b64 rc, {%6, %7};\n"
        "fma.rn.f32x2 rd, ra, rb, rc;\nmov.b64 {%0, %1}, rd;\n}\n"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 d;
    asm("{\n.reg .b64 ra, rb, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nmul.rn.f32x2 rd, ra, rb;\nmov.b64 {%0, %1}, rd;\n}\n"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 d;
    asm("{\n.reg .b64 ra, rb, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nadd.rn.f32x2 rd, ra, rb;\nmov.b64 {%0, %1}, rd;\n}\n"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float pow2i(int e) {                        // 2^e, e clamped to the normal range
    return __int_as_float((max(-126, min(127, e)) + 127) << 23);
}

// Byte offset of 16-byte chunk `chunk` (8 dims) of row `row` in an operand tile of fp16 rows: blocks of 64 dims, each
// [rows x 128 bytes] in the 128-byte swizzle pattern (8-row groups 1024 bytes apart).
__device__ __forceinline__ int op_off(int row, int chunk, int block_bytes) {
    return (chunk >> 3) * block_bytes + (row >> 3) * 1024 + (row & 7) * 128 + (((chunk & 7) ^ (row & 7)) << 4);
}
// Four int8 codes -> the same four integers as fp16.  The bytes become 1024 + (code + 128) as fp16 bit patterns
// (0x6400 | u8); subtracting 1152 is exact.
__device__ __forceinline__ void cvt4(uint32_t codes, uint32_t &lo, uint32_t &hi) {
    const uint32_t u = codes ^ 0x80808080u;
    lo = hsub2_u32(prmt(u, 0x64646464u, 0x4140u), 0x64806480u);
    hi = hsub2_u32(prmt(u, 0x64646464u, 0x4342u), 0x64806480u);
}
// Eight int4 codes (element 2j in the low nibble of byte j) -> fp16 pairs (0,1) (2,3) (4,5) (6,7).  A nibble becomes
// 1024 + (code + 8) as an fp16 bit pattern; subtracting 1032 is exact.
__device__ __forceinline__ void cvt8_i4(uint32_t w, uint32_t (&h)[4]) {
    uint32_t e[4];                                                     // elements (k, k + 4)
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = hsub2_u32(lop3_and_xor(w >> (4 * k), 0x000f000fu, 0x64086408u), 0x64086408u);
    h[0] = prmt(e[0], e[1], 0x5410u); h[1] = prmt(e[2], e[3], 0x5410u);
    h[2] = prmt(e[0], e[1], 0x7632u); h[3] = prmt(e[2], e[3], 0x7632u);
}
__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Block-32 rows: the power of two that a row's scales are multiplied with before they go into an fp16 operand.  Times any
// code the largest stays below the fp16 maximum if the scale does not exceed 2^12, and a scale of 2^-14 still has all its
// bits in the two limbs.  K rows: the largest finite scale to [2^11, 2^12).  V rows: the mean of the exponents to 2^-1,
// further down only for a scale beyond 2^12 times that: what is taken out of the operand rides in the row's weights, and
// with the largest scale there one outlier block left the other blocks' weights 2^-25 of ITS size (scales 2^16 apart:
// errors of 1e-2).  `nonfinite`: some block's scale is infinite or NaN (not counted).
template <int NBW>
__device__ __forceinline__ int b32_shift(const uint32_t (&w)[NBW], bool v, bool &nonfinite) {
    uint32_t m = 0, sum = 0, over = 0;                                 // of exponents + 1, both halves of a word; infinities and NaNs run over
#pragma unroll
    for (int i = 0; i < NBW; ++i) {
        const uint32_t x = (w[i] & 0x7fff7fffu) + 0x04000400u, e = (x >> 10) & 0x001f001fu;
        m = max_u16x2(m, e);
        sum += e;
        over |= x & 0x80008000u;
    }
    nonfinite = over != 0;
    const int most = 27 - max(2, (int)max(m & 0xffffu, m >> 16));
    return v ? min(most, 15 - (int)(((sum & 0xffffu) + (sum >> 16)) / (2 * NBW))) : most;
}
// Block-32 caches whose value scales overflowed fp16 (the codec stores infinity for blocks beyond 7 x 65504): adds such
// blocks to the output rows whose keys include them; any weight leaves code x infinity what it is.  Called by the softmax
// warps on the rows and dims each of their threads wrote.  Rare: one key at a time, out of line, and the CTA's place worked
// out again (in line, its registers cost the loops 84.9 -> 87.5 us for 2048 positions at head_dim 128; so 85.7).
template <int HD, int DV, int NQ>
__device__ __noinline__ void add_nonfinite_values(const PParams &p) {
    int bid;
    asm volatile("mov.u32 %0, %%ctaid.x;\n" : "=r"(bid));
    const int dpart = bid % (HD / DV);
    bid /= HD / DV;
    const int kvh = bid % p.nkv;
    bid /= p.nkv;
    const int b = bid % p.batch, tile = (p.q_blocks - 1 - bid / p.batch) * NQ + (NQ == 2 ? threadIdx.x >> 8 : 0);
    const int lane = threadIdx.x & 31, first_row = 32 * ((threadIdx.x >> 5) & 3) + 16 * ((threadIdx.x >> 7) & 1) + (lane >> 2);
#pragma unroll 1
    for (int row = first_row; row < first_row + 16; row += 8) {
        const int pos = tile * p.pos_per_tile + row / p.kvg;
        if (row >= p.pos_per_tile * p.kvg || pos >= p.S) continue;
        const int hi = min(p.d0 + pos, p.key_len - 1), lo = p.window > 0 ? max(0, p.d0 + pos - p.window + 1) : 0;
        const long at = b * p.out_batch_stride + ((long)pos * p.nh + kvh * p.kvg + row % p.kvg) * HD + dpart * DV + 2 * (lane & 3);
#pragma unroll 1
        for (int key = lo; key <= hi; ++key) {
            int slot = p.row0 + key;
            if (slot >= p.cache_cap) slot -= p.cache_cap;
            const size_t cr = (size_t)kvh * p.cache_cap + slot;
            const __half *scales = reinterpret_cast<const __half *>(p.v_scales + b * p.scale_batch_stride) + cr * (HD / 32) + dpart * (DV / 32);
            const uint8_t *codes = p.v_cache + b * p.kv_batch_stride + cr * p.row_bytes + dpart * (DV / 2) + (lane & 3);
#pragma unroll 1
            for (int c = 0; c < DV / 32; ++c) {
                const float sf = __half2float(scales[c]);
                if (isfinite(sf)) continue;
                for (int e = 0; e < 4; ++e) {
                    const int byte = codes[16 * c + 4 * e];
                    const float x = (float)nib_sext(byte & 15) * sf, y = (float)nib_sext(byte >> 4) * sf;
                    const long d = at + 32 * c + 8 * e;
                    if (p.out_type == ET_BF16) {
                        __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(reinterpret_cast<__nv_bfloat16 *>(p.out) + d);
                        *o = __floats2bfloat162_rn(__low2float(*o) + x, __high2float(*o) + y);
                    } else {
                        float2 *o = reinterpret_cast<float2 *>(reinterpret_cast<float *>(p.out) + d);
                        *o = make_float2(o->x + x, o->y + y);
                    }
                }
            }
        }
    }
}

template <int HD, int FMT, int QL, int NQ>
__global__ void __launch_bounds__(Cfg<HD, FMT, QL, NQ>::NTHREADS, 1) attn_prefill_kernel(const __grid_constant__ PParams p) {
    using C = Cfg<HD, FMT, QL, NQ>;
    constexpr int NSB = C::NSB, NSLOT = C::NSLOT, KL = C::KL, DV = C::DV, NCONST = C::NCONST;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *sm = smem_raw;
    const uint32_t sm_u32 = smem_u32(sm);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(sm + C::OFF_MISC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + C::OFF_MISC + 4);
    volatile int *v_nonfinite = reinterpret_cast<volatile int *>(sm + C::OFF_MISC + 8);       // block-32: some value block's scale is infinite or NaN
    const uint32_t bar0 = sm_u32 + C::OFF_BAR;
    auto bar_full = [&](int s) { return bar0 + 8 * s; };                          // dequant warps -> MMA
    auto bar_empty = [&](int s) { return bar0 + 8 * (NSLOT + s); };               // commit after the slot's last product -> dequant
    auto bar_const = [&](int i) { return bar0 + 8 * (2 * NSLOT + i); };           // dequant warps -> softmax: a tile's per-key constants
    auto bar_s_full = [&](int i) { return bar0 + 8 * (2 * NSLOT + NCONST + i); }; // commit after QK -> softmax
    auto bar_p_full = [&](int i) { return bar0 + 8 * (2 * NSLOT + NCONST + NSB + i); };      // softmax warps -> MMA
    auto bar_o_done = [&](int i) { return bar0 + 8 * (2 * NSLOT + NCONST + 2 * NSB + i); };  // commit after PV -> softmax (index: S buffer)
    const uint32_t bar_q_ready = bar0 + 8 * (2 * NSLOT + NCONST + 3 * NSB);       // softmax warps -> MMA

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // one-dimensional grid, heaviest work first: late query blocks (the most key tiles) of every KV head before earlier ones
    int bid = blockIdx.x;
    const int dpart = C::DSPLIT > 1 ? bid % C::DSPLIT : 0;
    bid /= C::DSPLIT;
    const int kvh = bid % p.nkv;
    bid /= p.nkv;
    const int b = bid % p.batch, qb = p.q_blocks - 1 - bid / p.batch;

    // key range of each query tile (whole key tiles), and of the CTA
    TileRange range[NQ];                               // tiles of query tile g, relative to the CTA's first (empty: first > last)
    int tile_lo = 0x7fffffff, tile_hi = -1;
#pragma unroll
    for (int g = 0; g < NQ; ++g) {
        const int s_first = (qb * NQ + g) * p.pos_per_tile;
        const int s_last = min(p.S, s_first + p.pos_per_tile) - 1;
        const int hi = s_last >= s_first ? min(p.d0 + s_last, p.key_len - 1) : -1;
        const int lo = p.window > 0 ? max(0, p.d0 + s_first - p.window + 1) : 0;
        if (hi >= lo) {
            range[g] = TileRange{lo / KT, hi / KT};
            tile_lo = min(tile_lo, range[g].first); tile_hi = max(tile_hi, range[g].last);
        } else {
            range[g] = TileRange{0x3fffffff, -1};
        }
    }
    const int n_tiles = tile_hi >= 0 ? tile_hi - tile_lo + 1 : 0;
    if (n_tiles == 0) tile_lo = 0;
#pragma unroll
    for (int g = 0; g < NQ; ++g) { range[g].first -= tile_lo; range[g].last -= tile_lo; }
    // (consecutive query tiles have overlapping or adjacent ranges, so every tile of the CTA serves at least one of them;
    // a tile that serves none, possible only with a window shorter than a query tile's span, costs its slots and no products)

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        *v_nonfinite = 0;
        for (int s = 0; s < NSLOT; ++s) { fused::mbar_init(bar_full(s), 2); fused::mbar_init(bar_empty(s), 1); }
        for (int i = 0; i < NCONST; ++i) fused::mbar_init(bar_const(i), 2);
        for (int i = 0; i < NSB; ++i) { fused::mbar_init(bar_s_full(i), 1); fused::mbar_init(bar_p_full(i), 8); fused::mbar_init(bar_o_done(i), 1); }
        fused::mbar_init(bar_q_ready, C::NSW);
        fused::fence_mbar_init();
    }
    if (warp == C::W_MMA) {
        tc5::tmem_alloc(sm_u32 + C::OFF_MISC, 512);
        tc5::tmem_relinquish();
    }
    tc5::tc_fence_before();
    __syncthreads();
    tc5::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    fused::pdl_wait();                         // the query and the cache rows may come from the stream predecessor
    fused::pdl_launch_dependents();

    if (warp == C::W_MMA) {
        // =========================================================== MMA issuer: one elected lane walks the schedule
        if (elect_one()) {
        constexpr uint32_t idesc_qk = make_idesc_f16(KT, false), idesc_pv = make_idesc_f16(128, true);
        const uint64_t qdesc = tc5::smem_desc_sw128(sm_u32 + C::OFF_Q);
        const uint64_t rdesc = tc5::smem_desc_sw128(sm_u32 + C::OFF_RING);
        // V operand, MN-major: the two 64-dim blocks of a slot are one operand, the second BLOCK bytes after the first
        // (leading-dimension offset); key groups of 8 rows stay 1024 bytes apart
        const uint64_t vrdesc = (rdesc & ~(0x3fffull << 16)) | ((uint64_t)(C::BLOCK >> 4) << 16);
        // the next unit of the ring: its first slot (a unit's KL slots share one pair of barriers, the first slot's)
        int ring = 0;
        uint32_t ring_phase = 0;
        auto next_unit = [&](int &slot) {
            slot = ring;
            const bool ok = wait_or_abort(bar_full(ring), ring_phase, abort_flag, p.fault);
            tc5::tc_fence_after();
            ring += KL;
            if (ring == NSLOT) { ring = 0; ring_phase ^= 1u; }
            return ok;
        };
        // S buffer buf += dims 128 c .. 128 c + 127 of query tile g x the K slots from n on
        auto qk = [&](int g, int buf, int c, int n) {
            const uint32_t d = tmem_base + C::TMEM_S + buf * KT;
#pragma unroll
            for (int kl = 0; kl < KL; ++kl) {
                const uint64_t bd = rdesc + (uint64_t)((n + kl) * (C::SLOT >> 4));
#pragma unroll
                for (int ql = 0; ql < QL; ++ql) {
                    if (ql + kl > 1) continue;                         // low x low: 2^-18 of the logit's terms and less
                    const uint64_t ad = qdesc + (uint64_t)(((g * QL + ql) * C::Q_LIMB + 2 * c * C::Q_BLOCK) >> 4);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_f16(d, ad + (uint64_t)(((k >> 2) * C::Q_BLOCK >> 4) + (k & 3) * 2), bd + (uint64_t)(((k >> 2) * C::BLOCK >> 4) + (k & 3) * 2),
                                 idesc_qk, (c | kl | ql | k) != 0 ? 1u : 0u);
                }
            }
        };
        // dims 128 c .. of O of query tile g += P in S buffer buf x the V slots from n on
        auto pv = [&](int g, int buf, int c, int n, bool first) {
            const uint32_t a = tmem_base + C::TMEM_S + buf * KT;
#pragma unroll
            for (int kl = 0; kl < KL; ++kl) {
                const uint64_t bd = vrdesc + (uint64_t)((n + kl) * (C::SLOT >> 4));
#pragma unroll
                for (int pl = 0; pl < 2; ++pl) {
                    if (pl + kl > 1) continue;
#pragma unroll
                    for (int k = 0; k < KT / 16; ++k)                  // 16 keys: 8 columns of A, 2048 bytes of the MN-major blocks
                        umma_f16_ts(tmem_base + C::TMEM_O + g * DV + c * 128, a + 32 * pl + 8 * k, bd + (uint64_t)(k * (2048 >> 4)),
                                    idesc_pv, (!first || kl || pl || k) ? 1u : 0u);
                }
            }
        };
        auto wait_bar = [&](uint32_t bar, uint32_t parity) {
            const bool ok = wait_or_abort(bar, parity, abort_flag, p.fault);
            tc5::tc_fence_after();
            return ok;
        };
        if (n_tiles > 0 && wait_bar(bar_q_ready, 0)) {
            struct Ops {
                decltype(next_unit) &next;
                decltype(wait_bar) &wait;
                decltype(qk) &qk_;
                decltype(pv) &pv_;
                decltype(bar_empty) &empty;
                decltype(bar_s_full) &s_full;
                decltype(bar_p_full) &p_full;
                decltype(bar_o_done) &od;
                __device__ __forceinline__ bool next_unit(int &slot) { return next(slot); }
                __device__ __forceinline__ void release(int slot) { tc5::umma_commit(empty(slot)); }
                __device__ __forceinline__ bool weights(int buf, int parity) { return wait(p_full(buf), parity); }
                __device__ __forceinline__ bool product(int buf, int parity) { return wait(od(buf), parity); }
                __device__ __forceinline__ void qk(int g, int buf, int c, int slot) { qk_(g, buf, c, slot); }
                __device__ __forceinline__ void s_done(int buf) { tc5::umma_commit(s_full(buf)); }
                __device__ __forceinline__ void pv(int g, int buf, int c, int slot, bool first) { pv_(g, buf, c, slot, first); }
                __device__ __forceinline__ void o_done(int buf) { tc5::umma_commit(od(buf)); }
            } ops{next_unit, wait_bar, qk, pv, bar_empty, bar_s_full, bar_p_full, bar_o_done};
            walk_products<NQ, HD / 128, DV / 128>(n_tiles, range, ops);
        }
        }
        __syncwarp();
    } else if (warp >= C::W_DEQ) {
        // =========================================================== dequant warps: cache bytes -> fp16 operand slots
        const int team = (warp - C::W_DEQ) >> 1, t = (threadIdx.x - 32 * C::W_DEQ) & 63;
        const uint8_t *gk = p.k_cache + b * p.kv_batch_stride, *gv = p.v_cache + b * p.kv_batch_stride;
        const uint8_t *gks = p.k_scales + b * p.scale_batch_stride, *gvs = p.v_scales + b * p.scale_batch_stride;
        // cache row of key index key (clamped into the array: masked keys then hold finite codes)
        auto cache_row = [&](int key) {
            int slot = p.row0 + max(0, min(key, p.key_len - 1));
            if (slot >= p.cache_cap) slot -= p.cache_cap;
            return (size_t)kvh * p.cache_cap + slot;
        };
        // piece k of this thread: 16-byte piece `ppc` of row prow + k * RSTEP of the slot.  Int8: the 8 lanes of a store
        // phase take 4 pieces of one 64-dim block from an even and from an odd row, whose swizzled chunks interleave (no
        // bank conflict).  RSTEP is a multiple of 8 rows: the swizzle is the same for every k
        const int prow = FMT == KV_I8 ? (t >> 5) * 4 + ((t >> 2) & 1) + 2 * ((t >> 4) & 1) : t >> 2;
        const int ppc = FMT == KV_I8 ? (t & 3) + 4 * ((t >> 3) & 1) : t & 3;
        constexpr int RSTEP = FMT == KV_I8 ? 8 : 16;
        static_assert(RSTEP % 8 == 0, "swizzle period");
        // byte offsets of the piece's 8-dim chunks inside a slot
        constexpr int NCH = C::CPP / 8;
        int soff[NCH];
#pragma unroll
        for (int e = 0; e < NCH; ++e) soff[e] = op_off(prow, NCH * ppc + e, C::BLOCK);
        auto unit_at = [&](int i) { return ring_unit<HD / 128, DV / 128>(i, n_tiles); };
        constexpr int NBW = C::NBW, NP = C::NP, TEAMS = C::TEAMS;
        constexpr int NSC = FMT == KV_I4B32 ? NP : 1, NCW = FMT == KV_I4B32 ? NBW : 1;
        // cache bytes of the team's next unit; with the first K unit of a tile the scales of key t of the tile
        uint4 x[NP];
        uint32_t sc[NSC], ckw[NCW], cvw[NCW];
        auto fetch = [&](RingUnit u) {
            const uint8_t *base = u.v ? gv : gk;
            const int key0 = (tile_lo + u.tile) * KT;
            const int dim0 = (u.v ? dpart * DV : 0) + u.c * 128;       // first dim of the slot
            const uint8_t *col = base + (FMT == KV_I8 ? dim0 : dim0 / 2) + 16 * ppc;
            // block-32: the piece is one block; the word that holds its fp16 scale
            const uint8_t *scol = (u.v ? gvs : gks) + ((dim0 >> 5) + ppc) / 2 * 4;
            int slot = p.row0 + key0;
            if (slot >= p.cache_cap) slot -= p.cache_cap;
            if (key0 + KT <= p.key_len && slot + KT <= p.cache_cap) {  // a whole tile in consecutive rows
                const size_t cr = (size_t)kvh * p.cache_cap + slot + prow;
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    x[k] = __ldcg(reinterpret_cast<const uint4 *>(col + cr * p.row_bytes + (size_t)(k * RSTEP) * p.row_bytes));
                    if constexpr (FMT == KV_I4B32) sc[k] = __ldcg(reinterpret_cast<const uint32_t *>(scol + (cr + k * RSTEP) * (NBW * 4)));
                }
            } else {
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    const size_t cr = cache_row(key0 + prow + k * RSTEP);
                    x[k] = __ldcg(reinterpret_cast<const uint4 *>(col + cr * p.row_bytes));
                    if constexpr (FMT == KV_I4B32) sc[k] = __ldcg(reinterpret_cast<const uint32_t *>(scol + cr * (NBW * 4)));
                }
            }
            if (!u.v && u.c == 0) {
                const size_t cr = cache_row(key0 + t);
#pragma unroll
                for (int w = 0; w < NCW; ++w) {
                    ckw[w] = __ldcg(reinterpret_cast<const uint32_t *>(gks) + cr * NCW + w);
                    cvw[w] = __ldcg(reinterpret_cast<const uint32_t *>(gvs) + cr * NCW + w);
                }
            }
        };
        auto store_const = [&](int tile) {                 // per-key constants of the tile (block-32: with the shifts the conversion reads back)
            float *cc = reinterpret_cast<float *>(sm + C::OFF_CONST + (tile % NCONST) * C::CONST_BYTES);
            if constexpr (FMT == KV_I4B32) {
                bool k_bad, v_bad;
                const int sk = b32_shift(ckw, false, k_bad), sv = b32_shift(cvw, true, v_bad);
                if (v_bad) *v_nonfinite = 1;
                cc[t] = pow2i(-sk);
                cc[KT + t] = (float)(-sv);
                cc[2 * KT + t] = pow2i(sv);
            } else {
                // (a NaN goes in with the logit: masked keys lose it in the mask's select)
                const float v = __uint_as_float(cvw[0]), vs = fmaxf(fabsf(v), VS_MIN);
                cc[t] = __uint_as_float(ckw[0]);
                cc[KT + t] = v == v ? lg2f(vs) : v;
                cc[2 * KT + t] = 1.0f / vs;
                const uint32_t neg = __ballot_sync(0xffffffffu, v < 0.0f);
                if (lane == 0) reinterpret_cast<uint32_t *>(cc + 3 * KT)[t >> 5] = neg;
            }
            __syncwarp();
            if (lane == 0) tc5::mbar_arrive(bar_const(tile % NCONST));
        };
        static_assert(KT == 64, "a team's 64 threads take one key each");
        auto convert = [&](RingUnit u, int slot) {
            uint8_t *s0 = sm + C::OFF_RING + slot * C::SLOT;
            uint8_t *s1 = s0 + (KL - 1) * C::SLOT;
            const float *cc = reinterpret_cast<const float *>(sm + C::OFF_CONST + (u.tile % NCONST) * C::CONST_BYTES);
            // zero weight x infinity is not zero: rows that may not see a key would be lost to its value, so infinities and
            // NaNs among V's block scales become finite here and reach the rows that do see them in add_nonfinite_values.
            // (A K row's leave through the select that masks the logits.)
            const float most = u.v ? 4096.0f : CUDART_INF_F;
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int row = prow + k * RSTEP, koff = k * RSTEP * 128;
                const uint32_t w[4] = {x[k].x, x[k].y, x[k].z, x[k].w};
                if constexpr (FMT == KV_I8) {
                    uint4 y0, y1;
                    cvt4(w[0], y0.x, y0.y); cvt4(w[1], y0.z, y0.w);
                    cvt4(w[2], y1.x, y1.y); cvt4(w[3], y1.z, y1.w);
                    *reinterpret_cast<uint4 *>(s0 + soff[0] + koff) = y0;
                    *reinterpret_cast<uint4 *>(s0 + soff[1] + koff) = y1;
                } else {
                    uint32_t hi2 = 0, lo2 = 0;
                    if constexpr (FMT == KV_I4B32) {
                        const uint32_t bits = (ppc & 1) ? sc[k] >> 16 : sc[k] & 0xffffu;        // (slots start at even blocks)
                        // the row's power of two: 1 / logit factor for K, 1 / value scale for V
                        const float up = u.v ? cc[2 * KT + row] : __uint_as_float(0x7f000000u - __float_as_uint(cc[row]));
                        const float sf = fmaxf(fminf(__half2float(__ushort_as_half((unsigned short)bits)) * up, most), -most);
                        const float sh = __uint_as_float(__float_as_uint(sf) & 0xfffe0000u);       // top 7 significant bits
                        hi2 = pack_f16x2(sh, sh);
                        lo2 = pack_f16x2(sf - sh, sf - sh);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        uint32_t h[4];
                        cvt8_i4(w[e], h);
                        const int off = soff[e] + koff;
                        if constexpr (FMT == KV_I4B32) {
                            *reinterpret_cast<uint4 *>(s0 + off) = make_uint4(hmul2_u32(h[0], hi2), hmul2_u32(h[1], hi2), hmul2_u32(h[2], hi2), hmul2_u32(h[3], hi2));
                            *reinterpret_cast<uint4 *>(s1 + off) = make_uint4(hmul2_u32(h[0], lo2), hmul2_u32(h[1], lo2), hmul2_u32(h[2], lo2), hmul2_u32(h[3], lo2));
                        } else {
                            *reinterpret_cast<uint4 *>(s0 + off) = make_uint4(h[0], h[1], h[2], h[3]);
                        }
                    }
                }
            }
        };
        const int n_units = n_tiles * ((HD + DV) / 128);
        auto wait_all = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag, p.fault)) != 0; };
        // this team's units are team, team + TEAMS, ...; its next one is on the way while the other teams' are converted
        RingUnit u = unit_at(team);
        if (team < n_units) fetch(u);
        for (int i = team; i < n_units; i += TEAMS) {
            const int n = i * KL, lap = n / NSLOT, slot = n - lap * NSLOT;
            if (lap > 0 && !wait_all(bar_empty(slot), (lap - 1) & 1)) break;
            if (!u.v && u.c == 0) store_const(u.tile);     // (behind the wait: see nconst)
            // (the shifts of the tile come from another thread, most often of another team)
            if (FMT == KV_I4B32 && !wait_all(bar_const(u.tile % NCONST), (u.tile / NCONST) & 1)) break;
            convert(u, slot);
            fused::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc5::mbar_arrive(bar_full(slot));
            if (i + TEAMS < n_units) {
                u = unit_at(i + TEAMS);
                fetch(u);
            }
        }
        __syncwarp();
    } else {
        // =========================================================== softmax warps
        const int g = NQ == 2 ? warp >> 3 : 0;
        const int half = (warp >> 2) & 1;                              // which 16 of the 32 lanes
        const uint32_t tmem_lane = tmem_base + ((uint32_t)(32 * (warp & 3) + 16 * half) << 16);
        const uint32_t tmem_o = tmem_lane + C::TMEM_O + g * DV;
        auto wait_warp = [&](uint32_t bar, uint32_t parity) {
            return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag, p.fault)) != 0;
        };
        // A warp works on 16 rows, a thread on two of them (8 q + lane / 4) and on every fourth pair of keys: a
        // key's constants cost a shared-memory read per two rows (a row per thread and three constants per key and row
        // took 1500 of the 4000 cycles of a 64-key step at head_dim 128 on the shared-memory port alone), and four softmax
        // warps per scheduler cover each other's waits and latencies (two, with 32 rows each: 3300 cycles per step)
        float qr[2], m[2];                       // logit factor, whole-number running reference
        F2 l[2];                                 // this thread's share of the denominator
        int all_lo = 0, all_hi = 0x7fffffff;     // keys that every row of the warp sees
        const int row0 = 16 * half + (lane >> 2);                      // of the quadrant's 32
        auto position = [&](int q) { return (qb * NQ + g) * p.pos_per_tile + (32 * (warp & 3) + row0 + 8 * q) / p.kvg; };
        auto in_use = [&](int q) { return 32 * (warp & 3) + row0 + 8 * q < p.pos_per_tile * p.kvg && position(q) < p.S; };
        auto key_range = [&](int q, int &lo, int &hi) {                // inclusive
            const int sr = position(q);
            hi = 0x7fffffff; lo = 0;             // (rows not in use: zero queries, never stored, not worth masking for)
            if (in_use(q)) {
                hi = min(p.d0 + sr, p.key_len - 1);
                if (p.window > 0) lo = max(0, p.d0 + sr - p.window + 1);
            }
        };
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            qr[q] = 0.0f;
            m[q] = M_INIT;
            l[q] = F2{0.0f, 0.0f};
            int lo, hi;
            key_range(q, lo, hi);
            all_lo = max(all_lo, lo);
            all_hi = min(all_hi, hi);
        }
        all_lo = __reduce_max_sync(0xffffffffu, all_lo);
        all_hi = __reduce_min_sync(0xffffffffu, all_hi);
        // ---- the warp's query rows times the power of two that takes a row's maximum to [2^14, 2^15), as one or two fp16
        // limbs (which of the two types the rows have decides QL).  The lanes share a row (whole lines per load, four rows in
        // flight, a short loop): a thread per row, eight dims at a time, took 12 us at head_dim 128 and 29 us at 256 before
        // the first product
        {
            constexpr int DPL = HD / 32, RW = QL == 2 ? DPL : DPL / 2, RB = 4;          // dims and 32-bit words per lane; rows in flight
            const int base_row = 32 * (warp & 3) + 16 * half;
            auto load_rows = [&](int r0, uint32_t (&x)[RB][RW]) {
#pragma unroll
                for (int jj = 0; jj < RB; ++jj) {
                    const int row = base_row + r0 + jj, sp = (qb * NQ + g) * p.pos_per_tile + row / p.kvg;
                    const bool use = row < p.pos_per_tile * p.kvg && sp < p.S;
                    const long off = b * p.q_batch_stride + ((long)sp * p.nh + kvh * p.kvg + row % p.kvg) * HD + DPL * lane;
#pragma unroll
                    for (int c = 0; c < RW / 2; ++c) {
                        const uint2 v = use ? __ldcg(reinterpret_cast<const uint2 *>(p.q + off * (QL == 2 ? 4 : 2)) + c) : make_uint2(0u, 0u);
                        x[jj][2 * c] = v.x; x[jj][2 * c + 1] = v.y;
                    }
                }
            };
            uint32_t cur[RB][RW], nxt[RB][RW];
            load_rows(0, cur);
#pragma unroll 1
            for (int r0 = 0; r0 < 16; r0 += RB) {
                if (r0 + RB < 16) load_rows(r0 + RB, nxt);
#pragma unroll
                for (int jj = 0; jj < RB; ++jj) {
                    float x[DPL];
#pragma unroll
                    for (int d = 0; d < DPL; ++d)
                        x[d] = __uint_as_float(QL == 2 ? cur[jj][d % RW] : (d & 1) ? cur[jj][d / 2 % RW] & 0xffff0000u : cur[jj][d / 2 % RW] << 16);
                    float amax = 0.0f;
#pragma unroll
                    for (int d = 0; d < DPL; ++d) amax = fmaxf(amax, fabsf(x[d]));
                    amax = tc5::redux_max(amax);
                    const int ex = (int)(__float_as_uint(amax) >> 23);                 // biased exponent (0: a zero or denormal row)
                    const int sh = ex > 0 ? min(126, 14 + 127 - ex) : 0;
                    const float up = pow2i(sh);
                    if ((lane >> 2) == ((r0 + jj) & 7)) { if (r0 < 8) qr[0] = pow2i(-sh) * p.q_scale; else qr[1] = pow2i(-sh) * p.q_scale; }
                    uint8_t *qt = sm + C::OFF_Q + g * QL * C::Q_LIMB;
                    const int row = base_row + r0 + jj;
#pragma unroll
                    for (int c = 0; c < DPL / 4; ++c) {                // 4 dims = half a 16-byte chunk
                        const int d0 = DPL * lane + 4 * c;
                        const float x0 = x[4 * c] * up, x1 = x[4 * c + 1] * up, x2 = x[4 * c + 2] * up, x3 = x[4 * c + 3] * up;
                        const __half2 h0 = __floats2half2_rn(x0, x1), h1 = __floats2half2_rn(x2, x3);
                        uint8_t *dst = qt + op_off(row, d0 >> 3, C::Q_BLOCK) + (d0 & 4) * 2;
                        *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
                        if constexpr (QL == 2)
                            *reinterpret_cast<uint2 *>(dst + C::Q_LIMB) = make_uint2(pack_f16x2(x0 - __low2float(h0), x1 - __high2float(h0)),
                                                                                     pack_f16x2(x2 - __low2float(h1), x3 - __high2float(h1)));
                    }
                }
#pragma unroll
                for (int jj = 0; jj < RB; ++jj)
#pragma unroll
                    for (int c = 0; c < RW; ++c) cur[jj][c] = nxt[jj][c];
            }
            fused::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc5::mbar_arrive(bar_q_ready);
        }
        bool alive = true;
        const int first = NQ == 2 && g == 1 ? range[NQ - 1].first : range[0].first, last = NQ == 2 && g == 1 ? range[NQ - 1].last : range[0].last;
        for (int i = max(first, 0); alive && i <= last; ++i) {
            const int it = i - first;                                  // this row's tiles so far
            const int buf = C::NB * g + it % C::NB;
            const uint32_t ts = tmem_lane + C::TMEM_S + buf * KT;
            const float *cc = reinterpret_cast<const float *>(sm + C::OFF_CONST + (i % NCONST) * C::CONST_BYTES);
            // (the constants were stored before the K slots of the tile: this wait only orders the reads; it may not come
            // first, a query tile whose range starts late would meet an older phase of the barrier)
            if (!wait_warp(bar_s_full(buf), (it / C::NB) & 1)) { alive = false; break; }
            if (!wait_warp(bar_const(i % NCONST), (i / NCONST) & 1)) { alive = false; break; }
            tc5::tc_fence_after();
            const int t0 = (tile_lo + i) * KT;
            F2 u[2][KT / 8];                     // [row][pair e: keys 8 e + 2 (lane % 4) + {0, 1}]
            {
                uint32_t x[32];
                tmem_ld_frag64(ts, x);
                tc5::tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; ++e) asm volatile("" : "+r"(x[e]));          // no use above the wait
#pragma unroll
                for (int e = 0; e < KT / 8; ++e)
#pragma unroll
                    for (int q = 0; q < 2; ++q) u[q][e] = F2{__uint_as_float(x[4 * e + 2 * q]), __uint_as_float(x[4 * e + 2 * q + 1])};
            }
            const F2 *cc2 = reinterpret_cast<const F2 *>(cc) + (lane & 3);
            float cm[2] = {-CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
            for (int e = 0; e < KT / 8; ++e) {
                const F2 a = cc2[4 * e], d = cc2[KT / 2 + 4 * e];
#pragma unroll
                for (int q = 0; q < 2; ++q) u[q][e] = fma2(mul2(u[q][e], a), F2{qr[q], qr[q]}, d);
            }
            // rows outside their range see nothing of a key (a select, never a multiply); tiles inside every row's range
            // carry no masking instructions at all
            if (t0 < all_lo || t0 + KT - 1 > all_hi) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    int lo, hi;
                    key_range(q, lo, hi);
#pragma unroll
                    for (int e = 0; e < KT / 8; ++e) {
                        const int t = t0 + 8 * e + 2 * (lane & 3);
                        u[q][e].x = (t >= lo && t <= hi) ? u[q][e].x : -CUDART_INF_F;
                        u[q][e].y = (t + 1 >= lo && t + 1 <= hi) ? u[q][e].y : -CUDART_INF_F;
                    }
                }
            }
            bool moved = false;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
                for (int e = 0; e < KT / 8; ++e) cm[q] = fmaxf(cm[q], fmaxf(u[q][e].x, u[q][e].y));
                moved = moved || cm[q] > m[q] + LAZY;
            }
            if (__any_sync(0xffffffffu, moved)) {
                // the reference of some rows moves, by a whole power of two: denominator and output sums follow
                float alpha[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    cm[q] = fmaxf(cm[q], __shfl_xor_sync(0xffffffffu, cm[q], 1));
                    cm[q] = fmaxf(cm[q], __shfl_xor_sync(0xffffffffu, cm[q], 2));
                    const float m_new = cm[q] > m[q] + LAZY ? ceilf(cm[q]) : m[q];
                    alpha[q] = m_new == m[q] ? 1.0f : (m[q] - m_new < -126.0f ? 0.0f : pow2i((int)(m[q] - m_new)));
                    m[q] = m_new;
                    l[q].x *= alpha[q]; l[q].y *= alpha[q];
                }
                if (it > 0) {
                    if (!wait_warp(bar_o_done(C::NB * g + (it - 1) % C::NB), ((it - 1) / C::NB) & 1)) { alive = false; break; }
                    tc5::tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < DV / 32; ++c) {
                        uint32_t x[16];
                        tmem_ld_frag32(tmem_o + 32 * c, x);
                        tc5::tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) x[e] = __float_as_uint(__uint_as_float(x[e]) * alpha[(e >> 1) & 1]);
                        tmem_st_frag32(tmem_o + 32 * c, x);
                    }
                }
            }
            // weights, in place of S: hi limbs in the buffer's first 32 columns, lo limbs in the others (a warp's rows are
            // its own, and all of their S is in registers)
            const F2 minus1{-1.0f, -1.0f};
            uint32_t ph[16], pl[16];
#pragma unroll
            for (int e = 0; e < KT / 8; ++e) {
                const F2 iv = cc2[KT + 4 * e];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    F2 w = add2(u[q][e], F2{-m[q], -m[q]});
                    w = F2{ex2f(w.x), ex2f(w.y)};
                    l[q] = fma2(w, iv, l[q]);
                    const __half2 hh = __floats2half2_rn(w.x, w.y);
                    ph[2 * e + q] = *reinterpret_cast<const uint32_t *>(&hh);
                    w = fma2(F2{__low2float(hh), __high2float(hh)}, minus1, w);
                    pl[2 * e + q] = pack_f16x2(w.x, w.y);
                }
            }
            if constexpr (FMT != KV_I4B32) {
                // negative value scales (no codec here writes one): the sign goes on the weights, past the denominator
                const uint2 neg = *reinterpret_cast<const uint2 *>(cc + 3 * KT);
                if ((neg.x | neg.y) != 0) {
#pragma unroll
                    for (int e = 0; e < KT / 8; ++e) {
                        const uint32_t two = (e < 4 ? neg.x : neg.y) >> (8 * (e & 3) + 2 * (lane & 3));
                        const uint32_t sign = ((two & 1u) << 15) | ((two & 2u) << 30);
#pragma unroll
                        for (int q = 0; q < 2; ++q) { ph[2 * e + q] ^= sign; pl[2 * e + q] ^= sign; }
                    }
                }
            }
            tmem_st_pairs32(ts, ph);
            tmem_st_pairs32(ts + 32, pl);
            tmem_wait_st();
            tc5::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc5::mbar_arrive(bar_p_full(buf));
        }
        // ---- output: O / l (rows without any key are exact zeros, lib/batched_attn_gpu.mojo:329-409)
        const int mine = last >= max(first, 0) ? last - first + 1 : 0;
        // (the barrier's phase before that is known to be over: S of the last tile was issued once that PV was done)
        if (alive && mine > 0) alive = wait_warp(bar_o_done(C::NB * g + (mine - 1) % C::NB), ((mine - 1) / C::NB) & 1);
        if (alive) {
            tc5::tc_fence_after();
            float inv[2];
            long oi[2];
            bool vr[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float x = l[q].x + l[q].y;
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                x += __shfl_xor_sync(0xffffffffu, x, 2);
                inv[q] = x > 0.0f ? 1.0f / x : (x == x ? 0.0f : x);
                const int row = 32 * (warp & 3) + row0 + 8 * q;
                vr[q] = in_use(q);
                oi[q] = b * p.out_batch_stride + ((long)position(q) * p.nh + kvh * p.kvg + row % p.kvg) * HD + dpart * DV + 2 * (lane & 3);
            }
#pragma unroll 1
            for (int c = 0; c < DV / 32; ++c) {
                uint32_t o[16];
                if (mine > 0) {
                    tmem_ld_frag32(tmem_o + 32 * c, o);
                    tc5::tmem_wait_ld();
                } else {
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = 0u;
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (!vr[q]) continue;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float x = __uint_as_float(o[4 * e + 2 * q]) * inv[q], y = __uint_as_float(o[4 * e + 2 * q + 1]) * inv[q];
                        const long at = oi[q] + 32 * c + 8 * e;
                        if (p.out_type == ET_BF16) *reinterpret_cast<__nv_bfloat162 *>(reinterpret_cast<__nv_bfloat16 *>(p.out) + at) = __floats2bfloat162_rn(x, y);
                        else *reinterpret_cast<float2 *>(reinterpret_cast<float *>(p.out) + at) = make_float2(x, y);
                    }
                }
            }
        }
    }

    // ------------------------------------------------------------ tear-down
    tc5::tc_fence_before();
    __syncthreads();
    if (warp == C::W_MMA) tc5::tmem_dealloc(tmem_base, 512);
    if (FMT == KV_I4B32 && warp < C::NSW && *v_nonfinite && !*abort_flag)
        add_nonfinite_values<HD, DV, NQ>(p);
}

}  // namespace pf
}  // namespace nomos
