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
