"""Back-to-back launch chains on one stream, without host synchronisation in between.

The attention kernels are launched with programmatic stream serialization: a grid may be set up, run its
warming pass over the query and request settled cache rows while its stream predecessor is still writing.
These tests put real producers in front of it and check every step of the chain against the oracle:
  * the producer epilogue rewrites the query IN PLACE and appends the newest rows, then the tcgen05 kernel
    (and the mma.sync kernel) reads them -- one query buffer reused by every step;
  * a decode loop on ONE cache where every step's attention call carries its own fused append and sets
    NOMOS_ATTN_SETTLED_CACHE, so step i+1 must not stream the row step i is still storing;
  * the same loop with the append as a call of its own (it lets the attention grid start early and writes other rows
    to other slots in every step), linear caches, wrapped rings and paged caches.
"""
import numpy as np
import pytest
import torch

from nomos_nvfp4_b200 import ops
from tests._cases import KVCache, bf16_normal
from tests._gpu import DEV, dev, host, within

pytestmark = pytest.mark.gpu
TOL = 2e-3
PATHS = {"auto": 0, "mma_sync": ops.NO_TCGEN05, "tcgen05": ops.TCGEN05_ALWAYS}


@pytest.mark.parametrize("path", ["mma_sync", "tcgen05"])
@pytest.mark.parametrize("n_s", [1, 9])
def test_producer_rewrites_the_query_in_place_then_attention_reads_it(oracle, path, n_s):
    rng = np.random.default_rng(160 + n_s)
    nh, nkv, hd, T0, steps = 8, 4, 128, 3000, 6
    cap = T0 + steps * n_s
    c = KVCache("i8", nkv, cap, hd)
    k0, v0 = bf16_normal(rng, (T0, nkv, hd)), bf16_normal(rng, (T0, nkv, hd))
    c.append(k0, v0, 0)
    ck, cv, cks, cvs = dev(c.k), dev(c.v), dev(c.ks), dev(c.vs)
    qw = dev((1.0 + 0.1 * rng.standard_normal(hd)).astype(np.float32)); kw = dev(np.ones(hd, np.float32))
    raw_q = dev(rng.standard_normal((steps, n_s, nh, hd)).astype(np.float32) * np.float32(3.0))
    raw_k = dev(rng.standard_normal((steps, n_s, nkv, hd)).astype(np.float32))
    raw_v = dev(rng.standard_normal((steps, n_s, nkv, hd)).astype(np.float32))
    dq = torch.zeros((n_s, nh, hd), dtype=torch.float32, device=DEV)           # ONE query buffer for every step
    outs = torch.full((steps, n_s, nh, hd), -1e30, dtype=torch.float32, device=DEV)
    k_used = torch.zeros((steps, n_s, nkv, hd), dtype=torch.float32, device=DEV); v_used = torch.zeros_like(k_used)
    args = []
    for i in range(steps):
        klen = T0 + (i + 1) * n_s
        a = ops.make_args(q=dq, k_cache=ck, v_cache=cv, k_scales=cks, v_scales=cvs, out=outs[i], kv_fmt=ops.KV_I8, S=n_s,
                          nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd, cache_hd=hd, cache_cap=cap, klen=klen, softmax_scale=0.09,
                          flags=PATHS[path] | ops.SETTLED_CACHE)
        args.append(a)
    need = max(ops.attn_workspace_bytes(a) for a in args)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    for a in args:
        a.workspace, a.ws_bytes = ws.data_ptr(), need
    torch.cuda.synchronize()
    for i in range(steps):                                                     # no synchronisation inside the loop
        dq.copy_(raw_q[i])
        ops.kv_norm_rope_append(None, dq, qw, raw_k[i], raw_v[i], kw, ck, cv, cks, cvs, n_s=n_s, nh=nh, nkv=nkv, l_hd=hd,
                                l_kvd=nkv * hd, cache_cap=cap, cache_hd=hd, base_pos=T0 + i * n_s, theta=10000.0, rope_dim=hd,
                                kv_fmt=ops.KV_I8, k_out=k_used[i], v_out=v_used[i])
        ops.attn_fused(None, args[i])
    torch.cuda.synchronize()
    # what the producer made of each step's query: the same kernel run alone on a copy (it is deterministic)
    q_used = []
    for i in range(steps):
        t = raw_q[i].clone()
        ops.kv_norm_rope_append(None, t, qw, raw_k[i], raw_v[i], kw, None, None, None, None, n_s=n_s, nh=nh, nkv=nkv, l_hd=hd,
                                l_kvd=nkv * hd, cache_cap=0, cache_hd=hd, base_pos=T0 + i * n_s, theta=10000.0, rope_dim=hd,
                                kv_fmt=-1)
        torch.cuda.synchronize()
        q_used.append(host(t))
    got = host(outs)
    for i in range(steps):
        c.append(host(k_used[i]), host(v_used[i]), T0 + i * n_s)
        klen = T0 + (i + 1) * n_s
        want = oracle.attn_exact(q_used[i], c.k, c.v, c.ks, c.vs, c.kv_fmt, nh, nkv, hd, hd, cap, S=n_s, window=0,
                                 query_base_pos=klen - n_s, win_lo=0, softmax_scale=0.09)
        for r in range(n_s):
            ok, rel = within(got[i][r], want[r], TOL)
            assert ok, f"step {i} row {r}: {rel:.2e} x RMS"
    assert np.array_equal(host(ck).view(np.uint8), c.k.view(np.uint8)) and np.array_equal(host(cks), c.ks)


@pytest.mark.parametrize("path", list(PATHS))
@pytest.mark.parametrize("n_new", [1, 4])
def test_single_cache_fused_append_loop_with_settled_cache_flag(oracle, path, n_new):
    """Every step appends its own rows inside the attention launch and declares the older rows settled; the next
    step's early reads must leave out the rows this step is still storing."""
    rng = np.random.default_rng(170 + n_new)
    nh, nkv, hd, steps = 8, 4, 128, 10
    T0 = 128 * 9 - 3                       # the appended rows cross a tile boundary during the loop
    cap = T0 + steps * n_new
    c = KVCache("i8", nkv, cap, hd)
    c.append(bf16_normal(rng, (T0, nkv, hd)), bf16_normal(rng, (T0, nkv, hd)), 0)
    ck, cv, cks, cvs = dev(c.k), dev(c.v), dev(c.ks), dev(c.vs)
    q = bf16_normal(rng, (steps, n_new, nh, hd))
    nk = bf16_normal(rng, (steps, n_new, nkv, hd)); nv = bf16_normal(rng, (steps, n_new, nkv, hd))
    dq, dnk, dnv = dev(q), dev(nk), dev(nv)
    outs = torch.full((steps, n_new, nh, hd), -1e30, dtype=torch.float32, device=DEV)
    args = []
    for i in range(steps):
        klen = T0 + (i + 1) * n_new
        args.append(ops.make_args(q=dq[i], k_cache=ck, v_cache=cv, k_scales=cks, v_scales=cvs, out=outs[i], kv_fmt=ops.KV_I8,
                                  S=n_new, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd, cache_hd=hd, cache_cap=cap, klen=klen,
                                  softmax_scale=0.1, new_k=dnk[i], new_v=dnv[i], n_new=n_new, new_base_pos=klen - n_new,
                                  flags=PATHS[path] | ops.SETTLED_CACHE))
    need = max(ops.attn_workspace_bytes(a) for a in args)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    for a in args:
        a.workspace, a.ws_bytes = ws.data_ptr(), need
    torch.cuda.synchronize()
    for a in args:
        ops.attn_fused(None, a)
    torch.cuda.synchronize()
    got = host(outs)
    for i in range(steps):
        c.append(nk[i], nv[i], T0 + i * n_new)
        klen = T0 + (i + 1) * n_new
        want = oracle.attn_exact(q[i], c.k, c.v, c.ks, c.vs, c.kv_fmt, nh, nkv, hd, hd, cap, S=n_new, window=0,
                                 query_base_pos=klen - n_new, win_lo=0, softmax_scale=0.1)
        for r in range(n_new):
            ok, rel = within(got[i][r], want[r], TOL)
            assert ok, f"step {i} row {r}: {rel:.2e} x RMS"
    assert np.array_equal(host(ck).view(np.uint8), c.k.view(np.uint8)) and np.array_equal(host(cks), c.ks)


@pytest.mark.parametrize("fmt,hd,nh,nkv,path", [("i8", 128, 8, 4, "mma_sync"), ("i8", 128, 8, 4, "tcgen05"), ("i4", 256, 4, 2, "auto"), ("i4b32", 256, 8, 4, "auto"),
                                               ("i4b32", 512, 8, 2, "auto")])
@pytest.mark.parametrize("n_s,window", [(1, 0), (9, 0), (1, 300), (9, 300)])
def test_append_call_then_attention_loop_with_settled_cache_flag(oracle, fmt, hd, nh, nkv, path, n_s, window):
    """append, attention, append, attention, ... without synchronisation: the append releases the attention grid before it
    has written a byte, and step i + 1's append must not overwrite a ring slot that step i still reads."""
    rng = np.random.default_rng(180 + n_s + hd + window)
    steps, T0 = 10, 1149
    cap = window + n_s - 1 if window else T0 + steps * n_s
    c = KVCache(fmt, nkv, cap, hd)
    first = max(0, T0 - cap) if window else 0
    c.append(bf16_normal(rng, (T0 - first, nkv, hd)), bf16_normal(rng, (T0 - first, nkv, hd)), first)
    ck, cv, cks, cvs = dev(c.k), dev(c.v), dev(c.ks), dev(c.vs)
    q = bf16_normal(rng, (steps, n_s, nh, hd))
    nk, nv = bf16_normal(rng, (steps, n_s, nkv, hd)), bf16_normal(rng, (steps, n_s, nkv, hd))
    dq, dnk, dnv = dev(q), dev(nk), dev(nv)
    outs = torch.full((steps, n_s, nh, hd), -1e30, dtype=torch.float32, device=DEV)
    args = []
    for i in range(steps):
        end = T0 + (i + 1) * n_s
        klen = min(cap, end)
        args.append(ops.make_args(q=dq[i], k_cache=ck, v_cache=cv, k_scales=cks, v_scales=cvs, out=outs[i], kv_fmt=c.kv_fmt, S=n_s, nh=nh, nkv=nkv, kvg=nh // nkv,
                                  l_hd=hd, cache_hd=hd, cache_cap=cap, win_start=end - klen, klen=klen, window=window, softmax_scale=0.1,
                                  flags=PATHS[path] | ops.SETTLED_CACHE))
    need = max(ops.attn_workspace_bytes(a) for a in args)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    for a in args:
        a.workspace, a.ws_bytes = ws.data_ptr(), need
    torch.cuda.synchronize()
    for i, a in enumerate(args):
        rows = (dnk[i], dnv[i], ck, cv, cks, cvs, n_s, nkv, hd, nkv * hd, cap, hd, T0 + i * n_s)
        if fmt == "i8":
            ops.gpu_append_quant_kv_i8(None, *rows)
        else:
            ops.gpu_append_quant_kv_i4(None, *rows, c.scale_blocks)
        ops.attn_fused(None, a)
    torch.cuda.synchronize()
    got = host(outs)
    for i in range(steps):
        c.append(nk[i], nv[i], T0 + i * n_s)
        end = T0 + (i + 1) * n_s
        want = oracle.attn_exact(q[i], c.k, c.v, c.ks, c.vs, c.kv_fmt, nh, nkv, hd, hd, cap, S=n_s, window=window, query_base_pos=end - n_s,
                                 win_lo=end - min(cap, end), softmax_scale=0.1)
        for r in range(n_s):
            ok, rel = within(got[i][r], want[r], TOL)
            assert ok, f"step {i} row {r}: {rel:.2e} x RMS"
    for d, h in ((ck, c.k), (cv, c.v), (cks, c.ks), (cvs, c.vs)):
        assert np.array_equal(host(d).view(np.uint8), h.view(np.uint8))


def test_paged_append_then_paged_attention_loop(oracle):
    rng = np.random.default_rng(190)
    nkv, hd, nh, steps, lens0 = 4, 128, 8, 10, [125, 300, 1200]
    page, per, batch = 128, 11, 3
    table = rng.permutation(batch * per).astype(np.int32).reshape(batch, per)
    caches = [KVCache("i8", nkv, per * page, hd) for _ in range(batch)]
    pools = np.zeros((2, batch * per, nkv, page, hd), np.int8)
    spools = np.ones((2, batch * per, nkv, page), np.float32)
    for b, (c, n) in enumerate(zip(caches, lens0)):
        c.append(bf16_normal(rng, (n, nkv, hd)), bf16_normal(rng, (n, nkv, hd)), 0)
        for j in range(per):
            at = slice(j * page, (j + 1) * page)
            pools[0, table[b, j]], pools[1, table[b, j]] = c.k[:, at], c.v[:, at]
            spools[0, table[b, j]], spools[1, table[b, j]] = c.row_scales_f32("k")[:, at], c.row_scales_f32("v")[:, at]
    q = bf16_normal(rng, (steps, batch, nh, hd))
    nk, nv = bf16_normal(rng, (steps, batch, nkv, hd)), bf16_normal(rng, (steps, batch, nkv, hd))
    dq, dnk, dnv, dt = dev(q), dev(nk), dev(nv), dev(table)
    kp, vp, ksp, vsp = dev(pools[0]), dev(pools[1]), dev(spools[0]), dev(spools[1])
    pos = dev(np.array([[n + i for n in lens0] for i in range(steps)], np.int32))
    lens = pos + 1
    outs = torch.full((steps, batch, nh, hd), -1e30, dtype=torch.float32, device=DEV)
    max_len = max(lens0) + steps
    wsb = ops.attn_paged_workspace_bytes(batch, nh, nkv, nh // nkv, hd, max_len)
    ws = torch.empty(max(wsb, 16), dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    for i in range(steps):
        ops.kv_paged_append_quant_i8(None, dnk[i], dnv[i], kp, vp, ksp, vsp, dt, pos[i], batch=batch, nkv=nkv, l_hd=hd, l_kvd=nkv * hd, max_pages=per)
        ops.attn_paged_decode_i8(None, dq[i], kp, vp, ksp, vsp, dt, lens[i], outs[i], ws, wsb, batch=batch, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd,
                                 n_pages=batch * per, max_pages=per, max_len=max_len, softmax_scale=0.1)
    torch.cuda.synchronize()
    got = host(outs)
    for i in range(steps):
        for b, c in enumerate(caches):
            n = lens0[b] + i
            c.append(nk[i, b][None], nv[i, b][None], n)
            want = oracle.attn_exact(q[i, b][None], c.k, c.v, c.ks, c.vs, c.kv_fmt, nh, nkv, hd, hd, per * page, S=1, query_base_pos=n, softmax_scale=0.1)
            ok, rel = within(got[i, b][None], want, TOL)
            assert ok, f"step {i} sequence {b}: {rel:.2e} x RMS"


@pytest.mark.parametrize("fmt,hd,nh,nkv,path", [("i8", 128, 8, 4, "mma_sync"), ("i8", 128, 8, 4, "tcgen05"), ("i4b32", 512, 8, 2, "auto")])
def test_a_long_append_holds_the_next_grid_back(oracle, fmt, hd, nh, nkv, path):
    """A chunk of 400 rows, then one query row that declares all but the newest two settled: the chunk's rows are there, not
    the ones that were in the cache before."""
    rng = np.random.default_rng(191 + hd)
    rounds, n_s = 6, 400
    c = KVCache(fmt, nkv, n_s, hd)
    ck, cv, cks, cvs = dev(c.k), dev(c.v), dev(c.ks), dev(c.vs)
    q = bf16_normal(rng, (rounds, 1, nh, hd))
    nk, nv = bf16_normal(rng, (rounds, n_s, nkv, hd)), bf16_normal(rng, (rounds, n_s, nkv, hd))
    dq, dnk, dnv = dev(q), dev(nk), dev(nv)
    outs = torch.full((rounds, 1, nh, hd), -1e30, dtype=torch.float32, device=DEV)
    args = [ops.make_args(q=dq[i], k_cache=ck, v_cache=cv, k_scales=cks, v_scales=cvs, out=outs[i], kv_fmt=c.kv_fmt, S=1, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd,
                          cache_hd=hd, cache_cap=n_s, klen=n_s, softmax_scale=0.1, flags=PATHS[path] | ops.SETTLED_CACHE) for i in range(rounds)]
    need = max(ops.attn_workspace_bytes(a) for a in args)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    for i, a in enumerate(args):
        a.workspace, a.ws_bytes = ws.data_ptr(), need
        rows = (dnk[i], dnv[i], ck, cv, cks, cvs, n_s, nkv, hd, nkv * hd, n_s, hd, 0)
        if fmt == "i8":
            ops.gpu_append_quant_kv_i8(None, *rows)
        else:
            ops.gpu_append_quant_kv_i4(None, *rows, c.scale_blocks)
        ops.attn_fused(None, a)
    torch.cuda.synchronize()
    got = host(outs)
    for i in range(rounds):
        c.append(nk[i], nv[i], 0)
        want = oracle.attn_exact(q[i], c.k, c.v, c.ks, c.vs, c.kv_fmt, nh, nkv, hd, hd, n_s, S=1, query_base_pos=n_s - 1, softmax_scale=0.1)
        ok, rel = within(got[i], want, TOL)
        assert ok, f"round {i}: {rel:.2e} x RMS"
