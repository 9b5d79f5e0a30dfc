"""The query-major prefill kernel over every cache format and head dim it serves, at the edges of its tiles: query tiles
of 128 rows (one or two per CTA at head_dim 128), key tiles of 64 keys, ragged ends, windows, wrapped rings, one and two
query limbs.  Checked against the oracle's fp64 attention over the same cache bytes.

Tolerance: 2e-4 x RMS per row for fp32 outputs.  The operands carry the codes, the block scales and bf16 queries exactly,
fp32 queries and weights to 2^-22 of the row's largest, so what is left is ex2.approx (2^-22), the rounding of logits of
about 100 to 2^-17 and of fp32 sums: a few 1e-5; bf16 outputs add their own rounding (2^-9 of the value, +1 ulp)."""
import numpy as np
import pytest
import torch

from nomos_nvfp4_b200 import ops
from tests._cases import KVCache, bf16_normal
from tests._gpu import DEV, dev, host, within
from tests.test_gpu_attn import build_cache
from tests.test_gpu_prefill import SENTINEL, run_fused

pytestmark = pytest.mark.gpu
TOL = 2e-4


def served(hd, q_type):
    return not (hd == 512 and q_type == ops.F32)


def check(oracle, c, q, got, *, S, klen, start, window, scale, bf16_out):
    nh = q.shape[-2]
    want = oracle.attn_exact(q, c.k, c.v, c.ks, c.vs, c.kv_fmt, nh, c.nkv, c.l_hd, c.cache_hd, c.cache_cap, S=S, window=window,
                             query_base_pos=start + klen - S, win_lo=start, softmax_scale=scale)
    assert not np.any(got == SENTINEL)
    for r in range(S):
        if bf16_out:
            tol = np.abs(want[r]) * 2.0 ** -8 + TOL * np.sqrt(np.mean(want[r] ** 2))
            assert np.all(np.abs(got[r] - want[r]) <= tol), f"row {r}"
        else:
            ok, rel = within(got[r], want[r], TOL)
            assert ok, f"row {r}: {rel:.2e} x RMS"


@pytest.mark.parametrize("q_type", [ops.F32, ops.BF16])
@pytest.mark.parametrize("hd", [128, 256, 512])
@pytest.mark.parametrize("fmt", ["i8", "i4", "i4b32"])
@pytest.mark.parametrize("S,klen,window,kvg", [(13, 13, 0, 2), (129, 129, 0, 1), (64, 321, 0, 4), (131, 259, 70, 2), (40, 513, 33, 8)])
def test_formats_and_head_dims(oracle, fmt, hd, q_type, S, klen, window, kvg):
    if not served(hd, q_type):
        pytest.skip("fp32 queries of 512-wide heads run as row groups")
    rng = np.random.default_rng(S + klen + hd + kvg)
    nkv = 2
    c = build_cache(fmt, rng, klen, nkv, hd, cap=klen + 3)
    q = bf16_normal(rng, (S, nkv * kvg, hd))
    scale = 1.0 / np.sqrt(hd)
    got, choice = run_fused(c, q, S=S, klen=klen, window=window, scale=scale, q_type=q_type, out_type=q_type, flags=ops.TCGEN05_ALWAYS)
    assert choice == 2
    check(oracle, c, q, got[0], S=S, klen=klen, start=0, window=window, scale=scale, bf16_out=q_type == ops.BF16)


@pytest.mark.parametrize("q_type", [ops.F32, ops.BF16])
@pytest.mark.parametrize("fmt", ["i8", "i4", "i4b32"])
@pytest.mark.parametrize("S,klen,window,kvg,nkv", [(576, 576, 0, 2, 16), (640, 640, 0, 2, 16), (129, 200, 0, 8, 20), (290, 430, 60, 4, 16)])
def test_one_and_two_query_tiles_per_cta(oracle, fmt, q_type, S, klen, window, kvg, nkv):
    """head_dim 128 on both sides of the size where CTAs take two query tiles (more tiles than the chip's 148 SMs: 144 in the
    first case, then 160, 180 with every head's last CTA half empty, 160); keys wrapped round the ring."""
    rng = np.random.default_rng(S + kvg)
    c = build_cache(fmt, rng, klen, nkv, 128, cap=klen + 5, start=klen + 9)
    q = bf16_normal(rng, (S, nkv * kvg, 128))
    scale = 1.0 / np.sqrt(128)
    got, choice = run_fused(c, q, S=S, klen=klen, win_start=klen + 9, window=window, scale=scale, q_type=q_type, out_type=q_type, flags=ops.TCGEN05_ALWAYS)
    assert choice == 2
    check(oracle, c, q, got[0], S=S, klen=klen, start=klen + 9, window=window, scale=scale, bf16_out=q_type == ops.BF16)


@pytest.mark.parametrize("hd,fmt,q_type", [(128, "i8", ops.F32), (128, "i4b32", ops.BF16), (256, "i4b32", ops.F32), (512, "i4", ops.BF16)])
def test_wrapped_ring(oracle, hd, fmt, q_type):
    """The window's keys run past the end of the ring: rows are addressed one by one."""
    rng = np.random.default_rng(hd)
    nkv, kvg, S, klen, start, cap, window = 2, 2, 90, 300, 1111, 333, 211
    c = build_cache(fmt, rng, klen, nkv, hd, cap=cap, start=start)
    q = bf16_normal(rng, (S, nkv * kvg, hd))
    scale = 1.0 / np.sqrt(hd)
    got, choice = run_fused(c, q, S=S, klen=klen, win_start=start, window=window, scale=scale, q_type=q_type, out_type=q_type, flags=ops.TCGEN05_ALWAYS)
    assert choice == 2
    check(oracle, c, q, got[0], S=S, klen=klen, start=start, window=window, scale=scale, bf16_out=q_type == ops.BF16)


@pytest.mark.parametrize("hd,fmt,q_type", [(128, "i8", ops.BF16), (128, "i4b32", ops.F32), (256, "i4", ops.BF16), (256, "i4b32", ops.F32), (512, "i4b32", ops.BF16), (512, "i8", ops.BF16)])
def test_batch_strides_and_a_wide_row_pitch(oracle, hd, fmt, q_type):
    """Two sequences with padded strides, cache rows wider than the head dim, and values of mean 2 (sums over all tiles)."""
    rng = np.random.default_rng(hd + 8)
    nkv, kvg, S, T, batch, cache_hd = 2, 2, 70, 203, 2, hd + 64
    nh, scale = nkv * kvg, 1.0 / np.sqrt(hd)
    cs = []
    for _ in range(batch):
        c = KVCache(fmt, nkv, T + 5, hd, cache_hd)
        c.append(bf16_normal(rng, (T, nkv, hd)), bf16_normal(rng, (T, nkv, hd)) + np.float32(2), 0)
        cs.append(c)
    q = bf16_normal(rng, (batch, S, nh, hd))

    def padded(arrays, pad):
        n = arrays[0].size * arrays[0].itemsize
        buf = np.full((len(arrays), n + pad), 0x55, np.uint8)
        for i, a in enumerate(arrays):
            buf[i, :n] = np.frombuffer(np.ascontiguousarray(a).tobytes(), np.uint8)
        return dev(buf), n + pad
    (k, kstride), (v, _) = padded([c.k for c in cs], 96), padded([c.v for c in cs], 96)
    (ks, sstride), (vs, _) = padded([c.ks for c in cs], 20), padded([c.vs for c in cs], 20)
    qs, os_ = S * nh * hd + 24, S * nh * hd + 40
    tt = torch.bfloat16 if q_type == ops.BF16 else torch.float32
    dq = torch.full((batch, qs), 7.0, dtype=tt, device=DEV)
    dq[:, :S * nh * hd] = dev(q.reshape(batch, -1)).to(tt)
    out = torch.full((batch, os_), SENTINEL, dtype=torch.float32, device=DEV)
    a = ops.make_args(q=dq, k_cache=k, v_cache=v, k_scales=ks, v_scales=vs, out=out, kv_fmt=cs[0].kv_fmt, q_type=q_type, out_type=ops.F32, batch=batch, S=S, nh=nh,
                      nkv=nkv, kvg=kvg, l_hd=hd, cache_hd=cache_hd, cache_cap=T + 5, klen=T, softmax_scale=scale, q_batch_stride=qs, out_batch_stride=os_,
                      kv_batch_stride=kstride, scale_batch_stride=sstride, flags=ops.TCGEN05_ALWAYS)
    assert ops.attn_kernel_choice(a) == 2
    ops.attn_fused(None, a)
    torch.cuda.synchronize()
    got = host(out)
    assert np.all(got[:, S * nh * hd:] == SENTINEL)
    for b, c in enumerate(cs):
        check(oracle, c, q[b], got[b, :S * nh * hd].reshape(S, nh, hd), S=S, klen=T, start=0, window=0, scale=scale, bf16_out=False)


@pytest.mark.parametrize("hd,fmt", [(256, "i8"), (256, "i4b32"), (512, "i4b32"), (512, "i4")])
def test_long_caches_and_values_of_one_sign(oracle, hd, fmt):
    """6000 keys in front of the chunk, values of mean 2: the fp32 sums of O run over a hundred tiles in tensor memory and no
    longer cancel.  T terms of one sign in fp32: T / 64 roundings of 2^-24 at the value's size, 6e-6 of it, within TOL."""
    rng = np.random.default_rng(hd + 9)
    nkv, kvg, S, T = 1, 4, 40, 6011
    c = KVCache(fmt, nkv, T, hd)
    c.append(bf16_normal(rng, (T, nkv, hd)), bf16_normal(rng, (T, nkv, hd)) + np.float32(2), 0)
    q, scale = bf16_normal(rng, (S, nkv * kvg, hd)), 1.0 / np.sqrt(hd)
    got, choice = run_fused(c, q, S=S, klen=T, scale=scale, q_type=ops.BF16, flags=ops.TCGEN05_ALWAYS)
    assert choice == 2
    check(oracle, c, q, got[0], S=S, klen=T, start=0, window=0, scale=scale, bf16_out=False)


@pytest.mark.parametrize("hd,fmt", [(128, "i8"), (256, "i4"), (512, "i4b32")])
def test_scales_far_apart(oracle, hd, fmt):
    """Rows, value rows and query rows whose magnitudes differ by up to 1e6 either way, and logits of thousands: the
    running reference moves often, and no limb may overflow or flush what matters."""
    rng = np.random.default_rng(900 + hd)
    nkv, kvg, S, T = 2, 2, 100, 400
    c = KVCache(fmt, nkv, T, hd)
    k, v = bf16_normal(rng, (T, nkv, hd)), bf16_normal(rng, (T, nkv, hd))
    lim = 3.0 if fmt == "i4b32" else 6.0             # block scales are fp16
    k *= np.float32(10.0) ** rng.uniform(-1, 1, (T, nkv, 1)).astype(np.float32)
    v *= np.float32(10.0) ** rng.uniform(-lim, lim, (T, nkv, 1)).astype(np.float32)
    c.append(k, v, 0)
    q = bf16_normal(rng, (S, nkv * kvg, hd)) * np.exp2(np.round(rng.uniform(-20, 6, (S, nkv * kvg, 1)))).astype(np.float32)
    got, choice = run_fused(c, q, S=S, klen=T, scale=1.0 / np.sqrt(hd), q_type=ops.BF16, flags=ops.TCGEN05_ALWAYS)
    assert choice == 2
    # logits reach several thousand here: their fp32 rounding (2^-12) moves the weights
    want = oracle.attn_exact(q, c.k, c.v, c.ks, c.vs, c.kv_fmt, nkv * kvg, nkv, hd, hd, T, S=S, query_base_pos=T - S, softmax_scale=1.0 / np.sqrt(hd))
    for r in range(S):
        ok, rel = within(got[0][r], want[r], 2e-3)
        assert ok, f"row {r}: {rel:.2e} x RMS"
    assert ops.device_faults() == 0


def test_a_row_of_infinities_stays_alone(oracle):
    """One query row is infinite, one NaN: the other rows of the same tile are what they are without them."""
    rng = np.random.default_rng(31)
    nkv, kvg, hd, S, T = 2, 2, 128, 64, 200
    c = build_cache("i8", rng, T, nkv, hd)
    q = bf16_normal(rng, (S, nkv * kvg, hd))
    clean, _ = run_fused(c, q, S=S, klen=T, scale=0.09)
    q[5, 1], q[9, 2, 3] = np.inf, np.nan
    got, _ = run_fused(c, q, S=S, klen=T, scale=0.09)
    keep = np.ones((S, nkv * kvg), bool)
    keep[5, 1] = keep[9, 2] = False
    assert np.array_equal(got[0][keep], clean[0][keep])


@pytest.mark.parametrize("q_type", [ops.F32, ops.BF16])
@pytest.mark.parametrize("hd", [128, 256, 512])
def test_an_infinite_value_block_reaches_only_the_rows_that_see_it(oracle, hd, q_type):
    """A block of one V row overflows its fp16 scale (or is infinite from the start): rows in front of the key and rows
    whose window has passed it are bit for bit what they are without it, the others lose that block's dims and no more."""
    if not served(hd, q_type):
        pytest.skip("fp32 queries of 512-wide heads run as row groups")
    rng = np.random.default_rng(hd + 5)
    nkv, kvg, S, T, window, key, blk = 2, 2, 150, 200, 40, 101, hd // 32 - 2
    k, v = bf16_normal(rng, (T, nkv, hd)), bf16_normal(rng, (T, nkv, hd))
    q, scale = bf16_normal(rng, (S, nkv * kvg, hd)), 1.0 / np.sqrt(hd)
    outs = []
    for bad in (False, True):
        c = KVCache("i4b32", nkv, T, hd)
        if bad:
            v[key, 0, 32 * blk:32 * blk + 32] *= np.float32(1e7)
            v[key, 1, 32 * blk + 3] = np.inf
        c.append(k, v, 0)
        if bad:                                        # codes of both signs under the infinite scale: infinities, not only NaNs
            c.v[0, key, 16 * blk:16 * blk + 4] = [0x71, 0xf0, 0x08, 0x9a]
        got, choice = run_fused(c, q, S=S, klen=T, window=window, scale=scale, q_type=q_type, out_type=q_type, flags=ops.TCGEN05_ALWAYS)
        assert choice == 2
        outs.append(got[0])
    rows = np.arange(S) + T - S
    sees = (rows >= key) & (rows < key + window)
    assert np.array_equal(outs[1][~sees], outs[0][~sees])
    want = oracle.attn_exact(q, c.k, c.v, c.ks, c.vs, c.kv_fmt, nkv * kvg, nkv, hd, hd, T, S=S, window=window, query_base_pos=T - S, softmax_scale=scale)
    dims = np.zeros(hd, bool)
    dims[32 * blk:32 * blk + 32] = True
    assert np.array_equal(outs[1][sees][..., dims], want[sees][..., dims], equal_nan=True) and not np.isfinite(want[sees][..., dims]).any()
    for r in np.flatnonzero(sees):
        if q_type == ops.BF16:
            assert np.all(np.abs(outs[1][r][:, ~dims] - want[r][:, ~dims]) <= np.abs(want[r][:, ~dims]) * 2.0 ** -8 + TOL)
        else:
            ok, rel = within(outs[1][r][:, ~dims], want[r][:, ~dims], TOL)
            assert ok, f"row {r}: {rel:.2e} x RMS"


@pytest.mark.parametrize("hd", [128, 256, 512])
def test_an_outlier_value_block_costs_the_other_blocks_nothing(oracle, hd):
    """One block of one V row is 2^16 times the others (its scale near the largest fp16): the row's other dims, where it adds
    nothing unusual, keep the accuracy of ordinary rows."""
    rng = np.random.default_rng(hd + 6)
    nkv, kvg, S, T, key, blk = 2, 2, 100, 300, 60, 1
    c = KVCache("i4b32", nkv, T, hd)
    k, v = bf16_normal(rng, (T, nkv, hd)), bf16_normal(rng, (T, nkv, hd))
    v[key, :, 32 * blk:32 * blk + 32] *= np.float32(2.0 ** 16)
    c.append(k, v, 0)
    q, scale = bf16_normal(rng, (S, nkv * kvg, hd)), 1.0 / np.sqrt(hd)
    got, choice = run_fused(c, q, S=S, klen=T, scale=scale, q_type=ops.BF16, flags=ops.TCGEN05_ALWAYS)
    assert choice == 2
    want = oracle.attn_exact(q, c.k, c.v, c.ks, c.vs, c.kv_fmt, nkv * kvg, nkv, hd, hd, T, S=S, query_base_pos=T - S, softmax_scale=scale)
    dims = np.zeros(hd, bool)
    dims[32 * blk:32 * blk + 32] = True
    for part in (dims, ~dims):
        for r in range(S):
            ok, rel = within(got[0][r][:, part], want[r][:, part], TOL)
            assert ok, f"row {r}: {rel:.2e} x RMS"


@pytest.mark.parametrize("hd,fmt", [(128, "i8"), (128, "i4"), (256, "i8"), (512, "i4")])
def test_negative_and_nan_value_scales(oracle, hd, fmt):
    """Row scales no codec here writes: negative ones multiply through like any other, a NaN one makes the rows that see its
    key NaN and no others."""
    rng = np.random.default_rng(hd + 7)
    nkv, kvg, S, T, key = 2, 2, 90, 260, 211
    c = build_cache(fmt, rng, T, nkv, hd)
    vs = c.vs.view(np.float32).reshape(nkv, T)
    vs *= np.where(rng.random((nkv, T)) < 0.3, np.float32(-1), np.float32(1))
    q, scale = bf16_normal(rng, (S, nkv * kvg, hd)), 1.0 / np.sqrt(hd)
    for nan in (False, True):
        if nan:
            vs[1, key] = np.nan
        got, choice = run_fused(c, q, S=S, klen=T, scale=scale, q_type=ops.BF16, flags=ops.TCGEN05_ALWAYS)
        assert choice == 2
        want = oracle.attn_exact(q, c.k, c.v, c.ks, c.vs, c.kv_fmt, nkv * kvg, nkv, hd, hd, T, S=S, query_base_pos=T - S, softmax_scale=scale)
        lost = np.isnan(want)
        assert lost.any() == nan and np.array_equal(np.isnan(got[0]), lost)
        for r in range(S):
            ok, rel = within(got[0][r][~lost[r]], want[r][~lost[r]], TOL)
            assert ok, f"row {r}: {rel:.2e} x RMS"


@pytest.mark.parametrize("hd,nh,nkv,fmt,S,klen,window,choice", [
    (256, 32, 16, "i8", 13, 2048, 0, 0), (256, 32, 16, "i8", 1024, 2048, 1024, 2), (256, 32, 16, "i4b32", 24, 16384, 0, 0),
    (512, 32, 4, "i4b32", 509, 4093, 0, 2), (512, 32, 4, "i8", 16, 16384, 0, 0), (128, 32, 16, "i4", 2048, 2048, 0, 2),
    (128, 8, 4, "i4b32", 40, 2048, 0, 0), (128, 8, 4, "i8", 40, 2048, 0, 2)])
def test_which_kernel_takes_a_prompt_chunk(hd, nh, nkv, fmt, S, klen, window, choice):
    """Few query rows against a long cache run as row groups with split keys, many on the query-major kernel."""
    a = ops.make_args(q=4096, k_cache=4096, v_cache=4096, k_scales=4096, v_scales=4096, out=4096, kv_fmt={"i8": ops.KV_I8, "i4": ops.KV_I4, "i4b32": ops.KV_I4B32}[fmt],
                      q_type=ops.BF16, out_type=ops.BF16, S=S, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd, cache_hd=hd, cache_cap=klen, klen=klen, window=window)
    assert ops.attn_kernel_choice(a) == choice


@pytest.mark.parametrize("nh,nkv,S,klen,window,choice", [
    (8, 4, 24, 16384, 0, 0), (32, 16, 24, 4096, 0, 0), (32, 16, 128, 4096, 0, 0), (32, 16, 256, 4096, 0, 2), (32, 16, 1024, 2048, 0, 2),
    (32, 8, 64, 16384, 0, 0), (32, 16, 64, 1088, 1024, 0), (32, 16, 1024, 2048, 1024, 2)])
def test_which_kernel_takes_a_prompt_chunk_on_a_wrapped_int8_ring(nh, nkv, S, klen, window, choice):
    cap = klen + 8
    a = ops.make_args(q=4096, k_cache=4096, v_cache=4096, k_scales=4096, v_scales=4096, out=4096, kv_fmt=ops.KV_I8, q_type=ops.BF16, out_type=ops.BF16,
                      S=S, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=128, cache_hd=128, cache_cap=cap, win_start=cap + cap // 2, klen=klen, window=window)
    assert ops.attn_kernel_choice(a) == choice
