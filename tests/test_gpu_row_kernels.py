"""The row kernels (appends, producer, window readers) and the streaming dense attention where their fast paths begin and
end: many tokens per launch, cache rows that are no whole 4-byte words, key counts around a warp's loads in flight."""
import numpy as np
import pytest
import torch

from nomos_nvfp4_b200 import ops
from tests._cases import KVCache, bf16_normal
from tests._gpu import DEV, dev, host
from tests.test_gpu_producer import run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,hd", [("i8", 128), ("i4", 256), ("i4b32", 512)])
def test_producer_many_tokens(fmt, hd):
    """700 tokens: one CTA per token, every warp walks several rows; odd head counts."""
    run_case(fmt, hd=hd, nh=3, nkv=3, n_s=700, base_pos=300, cap=768, theta=10000.0, rope_dim=hd // 4, seed=21)


@pytest.mark.parametrize("fmt", ["i8", "i4", "i4b32"])
@pytest.mark.parametrize("hd,cache_hd,n_s", [(128, 128, 67), (128, 132, 5), (256, 260, 3), (512, 520, 2), (64, 64, 4)])
def test_append_bytes_on_both_sides_of_the_register_kernel(fmt, hd, cache_hd, n_s):
    """Rows of whole 4-byte words and not, bit for bit against the oracle's codec (exact zeros and ties among the values)."""
    rng = np.random.default_rng(hd + cache_hd)
    nkv, cap, base = 3, 71, 68
    c = KVCache(fmt, nkv, cap, hd, cache_hd)
    k, v = bf16_normal(rng, (n_s, nkv, hd)), bf16_normal(rng, (n_s, nkv, hd))
    k[0, 0] = 0.0
    v[1, 1, ::3] = 3.5
    d = [dev(c.k), dev(c.v), dev(c.ks), dev(c.vs)]
    if fmt == "i8":
        ops.gpu_append_quant_kv_i8(None, dev(k), dev(v), *d, n_s, nkv, hd, nkv * hd, cap, cache_hd, base)
    else:
        ops.gpu_append_quant_kv_i4(None, dev(k), dev(v), *d, n_s, nkv, hd, nkv * hd, cap, cache_hd, base, c.scale_blocks)
    torch.cuda.synchronize()
    c.append(k, v, base)
    for got, want in zip(d, (c.k, c.v, c.ks, c.vs)):
        assert np.array_equal(host(got), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,T", [(4, 2, 128, 31), (4, 2, 128, 33), (8, 2, 128, 1027), (6, 2, 256, 517), (4, 2, 512, 63), (16, 16, 128, 4099)])
def test_dense_decode_key_counts(dtype, nh, nkv, hd, T):
    """fp32 sums in any order: within 1e-5 x RMS of 64 bits (logits of a few units, T terms of 2^-24 each)."""
    g = torch.Generator(device=DEV); g.manual_seed(T)
    k, v = (torch.randn(nkv, T + 5, hd, generator=g, device=DEV).to(dtype) for _ in range(2))
    q = torch.randn(nh, hd, generator=g, device=DEV) * hd ** -0.5
    scratch, out = torch.empty(nh * T, device=DEV), torch.full((nh, hd), -1e30, device=DEV)
    if dtype == torch.float32:
        ops.attention_gpu_fp32_dev(None, None, q, k, v, scratch, out, nh, nkv, hd, hd, T + 5, T, nh // nkv)
    else:
        ops.attention_gpu_bf16_dev(None, None, q, k, v, scratch, 0, 0, out, nh, nkv, hd, hd, T + 5, T, nh // nkv)
    kk, vv = (x[:, :T].double().repeat_interleave(nh // nkv, 0) for x in (k, v))
    want = (torch.softmax((q.double()[:, None] * kk).sum(-1), -1)[..., None] * vv).sum(1)
    assert (out.double() - want).abs().max().item() <= 1e-5 * want.square().mean().sqrt().item()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("S,T", [(1, 40), (1, 4099), (37, 400)])
def test_dense_a_nan_stays_one(dtype, S, T):
    """A NaN or infinite key: rows that see it are NaN whatever the number of splits, heads and rows that do not are bit for
    bit what they are without it."""
    g = torch.Generator(device=DEV); g.manual_seed(S + T)
    nh, nkv, hd, key = 4, 2, 128, T - (S + 1) // 2
    k, v = (torch.randn(nkv, T, hd, generator=g, device=DEV).to(dtype) for _ in range(2))
    q = torch.randn(S, nh, hd, generator=g, device=DEV) * hd ** -0.5
    scratch = torch.empty(S * nh * T, device=DEV)
    f = ops.attention_prefill_prefix_batched_fp32 if dtype == torch.float32 else ops.attention_prefill_prefix_batched_bf16
    outs = []
    for bad in (None, float("nan"), float("inf")):
        if bad is not None:
            k[0, key] = bad
        out = torch.full((S, nh, hd), -1e30, device=DEV)
        a = (q, 0, scratch, 0, out, k, v) if dtype == torch.float32 else (q, 0, 0, scratch, 0, 0, out, k, v)
        f(None, None, *a, nh, nkv, hd, hd, T, S, T, nh // nkv, 0, T - S, 0)
        outs.append(host(out))
    sees = np.zeros((S, nh), bool)
    sees[np.arange(S) + T - S >= key, :nh // nkv] = True
    for got in outs[1:]:
        assert np.array_equal(got[~sees], outs[0][~sees]) and np.isnan(got[sees]).all() and sees.any()


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("hd,shift", [(128, 0), (512, 0), (256, 8)])
def test_block32_reader_to_int8_every_code(oracle, hd, shift, special):
    """All 16 nibble values under scales from subnormal to large (special: also infinite and zero), aligned rows (table kernel) and rows 8 bytes off (general
    kernel): the same bytes from both, and the reference's arithmetic (multiply, divide, round away) in float32."""
    rng = np.random.default_rng(hd)
    nkv, cap, klen, start, nb = 2, 37, 29, 20, hd // 32
    codes = rng.integers(0, 256, (nkv, cap, hd // 2), dtype=np.uint8)
    s16 = (2.0 ** rng.uniform(-16, 6, (nkv, cap, nb))).astype(np.float16)
    if special:                                        # overflowed and empty blocks, rows of zeros
        s16[0, ::5, 0], s16[0, 1::5, 1], s16[1, ::7] = np.inf, 0, 0
    q8 = (s16.astype(np.float32).max(-1) * np.float32(7.0) / np.float32(127.0)).astype(np.float32)
    q8[q8 == 0] = 1
    scales = np.concatenate([s16.view(np.uint8).ravel(), q8.view(np.uint8).ravel()])
    raw = torch.zeros(codes.size + 64, dtype=torch.uint8, device=DEV)
    raw[shift:shift + codes.size] = dev(codes.ravel())
    out, osc = torch.zeros(nkv, klen, hd, dtype=torch.int8, device=DEV), torch.zeros(nkv, klen, device=DEV)
    ops.gpu_dequant_kv_i4_to_q8_layer(None, raw.data_ptr() + shift, dev(scales), out, osc, nkv, klen, hd, klen, cap, start, nb)
    torch.cuda.synchronize()
    slots = (start + np.arange(klen)) % cap
    nib = np.stack([codes & 15, codes >> 4], -1).reshape(nkv, cap, hd).astype(np.int32)
    q = ((nib ^ 8) - 8).astype(np.float32)
    with np.errstate(invalid="ignore"):
        x = (q * np.repeat(s16.astype(np.float32), 32, -1)) / q8[..., None]
        y = np.trunc(x + np.where(x >= 0, np.float32(0.5), np.float32(-0.5)).astype(np.float32))
    want = np.clip(np.where(np.isnan(y), 0, y), -127, 127).astype(np.int8)      # (a NaN converts to 0)
    assert np.array_equal(host(out), want[:, slots]) and np.array_equal(host(osc), q8[:, slots])
