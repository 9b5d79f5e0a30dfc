"""The work a user of this library has it do: one layer's attention calls over quantised and dense KV caches.

Kinds of case (`kind`):
  step     one decode or verify step: quantise the S newest K/V rows into the cache and attend them with everything
           before (nomos_attn_fused, the append fused into the launch or as its own call before it)
  paged    the same for a batch of sequences of different lengths on paged int8 caches
  prompt   a chunk of prompt positions behind a cached prefix: causal / sliding-window attention of many query rows,
           through the superset call or through the reference's prefix operator
  rows     the producer epilogue of a prompt chunk: norms, RoPE and quantise-on-write of many rows
  dense    the reference's unquantised fp32 / bf16 KV modes, one row or a chunk
Inputs are N(0,1) rows rounded to bf16, K with four outlier channels per head (x8), as the benchmark makes them.
"""
import math

import torch

from nomos_nvfp4_b200 import ops

DEV = "cuda"
FMT = {"i8": ops.KV_I8, "i4": ops.KV_I4, "i4b32": ops.KV_I4B32}
ET = {"bf16": ops.BF16, "fp32": ops.F32}
TT = {"bf16": torch.bfloat16, "fp32": torch.float32}


def listed():
    return [
        # the smallest call there is: a short chat's first tokens, where launches and latency are everything
        {"name": "decode_512_i8", "kind": "step", "fmt": "i8", "nh": 8, "nkv": 4, "hd": 128, "S": 1, "keys": 512, "window": 0, "append": "fused", "io": "bf16"},
        # a sliding-window layer of the model, wrapped ring, the new row quantised in the launch
        {"name": "decode_ring1024_i4b32_hd256", "kind": "step", "fmt": "i4b32", "nh": 32, "nkv": 16, "hd": 256, "S": 1, "keys": 8192, "window": 1024, "append": "fused", "io": "bf16"},
        # the headline: a global-attention layer at 32768 keys, int8
        {"name": "decode_32k_i8", "kind": "step", "fmt": "i8", "nh": 32, "nkv": 16, "hd": 128, "S": 1, "keys": 32768, "window": 0, "append": "fused", "io": "bf16"},
        # a full-attention layer of the model (4 KV heads of 512), append and attention as two calls
        {"name": "decode_32k_i4b32_hd512", "kind": "step", "fmt": "i4b32", "nh": 32, "nkv": 4, "hd": 512, "S": 1, "keys": 32768, "window": 0, "append": "call", "io": "bf16"},
        # speculative verify of nine draft tokens
        {"name": "verify9_16k_i8", "kind": "step", "fmt": "i8", "nh": 32, "nkv": 16, "hd": 128, "S": 9, "keys": 16393, "window": 0, "append": "call", "io": "bf16"},
        # batched serving on paged caches, every sequence of another length
        {"name": "paged_batch8_i8", "kind": "paged", "nh": 32, "nkv": 16, "batch": 8, "keys": 20011, "io": "bf16"},
        # a whole prompt on the configurations' geometry
        {"name": "prompt_2048_i8", "kind": "prompt", "fmt": "i8", "nh": 32, "nkv": 16, "hd": 128, "S": 2048, "keys": 2048, "window": 0, "io": "bf16", "api": "fused"},
        # a prompt chunk of a sliding-window layer the way the reference's engine runs it: int4 ring read out as int8
        # rows, then the fp32 prefix operator over them
        {"name": "chunk_1024_sliding_hd256", "kind": "prompt", "fmt": "i4b32", "nh": 32, "nkv": 16, "hd": 256, "S": 1024, "keys": 2047, "window": 1024, "io": "fp32", "api": "prefix"},
        # a ragged prompt chunk of a full-attention layer straight off the int4 cache
        {"name": "chunk_509_full_hd512", "kind": "prompt", "fmt": "i4b32", "nh": 32, "nkv": 4, "hd": 512, "S": 509, "keys": 4093, "window": 0, "io": "bf16", "api": "fused"},
        # the rows of a prompt chunk on their way into the cache
        {"name": "rows_2048_i4b32_hd256", "kind": "rows", "fmt": "i4b32", "nh": 32, "nkv": 16, "hd": 256, "S": 2048, "cap": 4096},
        # the unquantised modes: a decode step on a bf16 cache, and a chunk behind a prefix
        {"name": "dense_decode_8k_bf16", "kind": "dense", "kv": "bf16", "nh": 32, "nkv": 16, "hd": 128, "S": 1, "keys": 8192, "window": 0},
        {"name": "dense_chunk_256_bf16", "kind": "dense", "kv": "bf16", "nh": 32, "nkv": 16, "hd": 128, "S": 256, "keys": 2048, "window": 0},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of its range, odd or even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    geo = [(8, 4, 128), (32, 16, 128), (32, 8, 128), (16, 16, 128), (32, 16, 256), (32, 4, 512)]
    kind = rng.choice(["step", "step", "step", "paged", "prompt", "prompt", "rows", "dense"])
    nh, nkv, hd = rng.choice(geo)
    if kind == "step":
        s = rng.choice([1, 1, 1, 2, 5, 9])
        window = rng.choice([0, 0, 0, 1024, 512])
        fmt = rng.choice(["i8", "i8", "i4", "i4b32"])
        return {"kind": "step", "fmt": fmt, "nh": nh, "nkv": nkv, "hd": hd, "S": s, "keys": _size(rng, 300, 65536 if hd == 128 else 32768), "window": window,
                "append": rng.choice(["fused", "call"]), "io": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "paged":
        nh, nkv, _ = rng.choice(geo[:4])
        return {"kind": "paged", "nh": nh, "nkv": nkv, "batch": rng.randint(1, 8), "keys": _size(rng, 200, 20011), "io": rng.choice(["bf16", "fp32"])}
    if kind == "prompt":
        s = _size(rng, 24, 2048 if hd == 128 else 640)
        return {"kind": "prompt", "fmt": rng.choice(["i8", "i8", "i4", "i4b32"]), "nh": nh, "nkv": nkv, "hd": hd, "S": s,
                "keys": s + rng.choice([0, _size(rng, 1, 2048)]), "window": rng.choice([0, 0, 1024]), "io": rng.choice(["bf16", "fp32"]),
                "api": rng.choice(["fused", "prefix"])}
    if kind == "rows":
        return {"kind": "rows", "fmt": rng.choice(["i8", "i4", "i4b32"]), "nh": nh, "nkv": nkv, "hd": hd, "S": _size(rng, 1, 2048), "cap": 4096}
    s = rng.choice([1, _size(rng, 2, 256)])
    return {"kind": "dense", "kv": rng.choice(["bf16", "fp32"]), "nh": nh, "nkv": nkv, "hd": hd, "S": s,
            "keys": max(s, _size(rng, 300, 8192 if s == 1 else 2048)), "window": rng.choice([0, 0, 1024])}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device=DEV).to(torch.bfloat16).float()


def _rows(g, n, nkv, hd):
    """K and V rows [n, nkv, hd] fp32 as a projection leaves them."""
    k, v = _normal(g, n, nkv, hd), _normal(g, n, nkv, hd)
    gain = torch.ones((nkv, hd), device=DEV)
    gain.scatter_(1, torch.rand((nkv, hd), generator=g, device=DEV).argsort(1)[:, :4], 8.0)
    return k * gain, v


def _away(x, lim):
    return torch.trunc(x + torch.where(x >= 0, 0.5, -0.5)).clamp(-lim, lim)


def _quant(x, fmt):
    """Codes (float) and the scale of every element, of rows [..., hd]: the codecs' arithmetic in plain torch."""
    if fmt == "i4b32":
        b = x.unflatten(-1, (-1, 32))
        a = b.abs().amax(-1, keepdim=True)
        s = torch.where(a > 0, a / torch.full_like(a, 7.0), torch.ones_like(a)).half().float()
        return _away(b / s, 7).flatten(-2), s.expand_as(b).flatten(-2)
    lim = 127 if fmt == "i8" else 7
    a = x.abs().amax(-1, keepdim=True)
    s = a / torch.full_like(a, float(lim))
    s = torch.where(s == 0, torch.ones_like(s), s)
    return _away(x * (torch.ones_like(s) / s), lim), s.expand_as(x)


def _scale_bytes(fmt, nkv, cap, hd):
    return nkv * cap * (hd // 32 * 2 + 4 if fmt == "i4b32" else 4)


def _pack(x, fmt, cap, slots):
    """Cache plane and scale buffer holding the rows x [n, nkv, hd] at `slots` of a ring of `cap`."""
    n, nkv, hd = x.shape
    code, sc = _quant(x, fmt)
    code, sc = code.transpose(0, 1), sc.transpose(0, 1)
    if fmt == "i8":
        plane = torch.zeros((nkv, cap, hd), dtype=torch.int8, device=DEV)
        plane[:, slots] = code.to(torch.int8)
    else:
        nib = code.to(torch.int16) & 15
        plane = torch.zeros((nkv, cap, hd // 2), dtype=torch.uint8, device=DEV)
        plane[:, slots] = (nib[..., 0::2] | (nib[..., 1::2] << 4)).to(torch.uint8)
    buf = torch.zeros(_scale_bytes(fmt, nkv, cap, hd), dtype=torch.uint8, device=DEV)
    if fmt == "i4b32":
        nb = hd // 32
        fine, row = buf[: nkv * cap * nb * 2].view(torch.float16), buf[nkv * cap * nb * 2:].view(torch.float32)
        s16 = sc[..., ::32].half()
        fine.view(nkv, cap, nb)[:, slots] = s16
        q8 = (s16.float().amax(-1) * 7.0)
        row.view(nkv, cap)[:, slots] = q8 / torch.full_like(q8, 127.0)
    else:
        buf.view(torch.float32).view(nkv, cap)[:, slots] = sc[..., 0]
    return plane, buf


def _dequant(x, fmt):
    """What the cache makes of rows [n, nkv, hd], in 64 bits."""
    code, sc = _quant(x, fmt)
    return code.double() * sc.double()


def _via_q8(x):
    """Rows read out of a block-32 int4 cache as int8 rows: codes requantised to the cached row scale."""
    code, sc = _quant(x, "i4b32")
    q8 = sc.amax(-1, keepdim=True) * 7.0
    q8 = q8 / torch.full_like(q8, 127.0)
    return _away(code * sc / q8, 127).double() * q8.double()


def _attend(q, k, v, d0, window, scale):
    """Exact attention in 64 bits: q [S, nh, hd], k / v [T, nkv, hd]; row s sees keys [max(0, d0+s-window+1), d0+s]."""
    s, nh, hd = q.shape
    t, nkv, _ = k.shape
    out = torch.empty((s, nh, hd), dtype=torch.float64, device=DEV)
    q, k, v = q.double(), k.double(), v.double()
    hi = torch.arange(s, device=DEV)[:, None] + d0
    at = torch.arange(t, device=DEV)[None, :]
    seen = (at <= hi) & (at > hi - window) if window > 0 else at <= hi
    for h in range(nh):
        g = h // (nh // nkv)
        p = (q[:, h] @ k[:, g].T) * scale
        p = torch.softmax(p.masked_fill(~seen, -math.inf), -1)
        out[:, h] = p @ v[:, g]
    return out


def _step_span(c):
    """(ring capacity, window start, keys in the window) of a step whose newest row is position keys - 1."""
    if not c["window"]:
        return c["keys"] + 7 & ~7, 0, c["keys"]
    cap = c["window"] + c["S"] - 1
    klen = min(cap, c["keys"])
    return cap, c["keys"] - klen, klen


def _step_inputs(c, g):
    _, _, klen = _step_span(c)
    k, v = _rows(g, klen, c["nkv"], c["hd"])
    return k, v, _normal(g, c["S"], c["nh"], c["hd"])


def _prompt_inputs(c, g):
    k, v = _rows(g, c["keys"], c["nkv"], c["hd"])
    return k, v, _normal(g, c["S"], c["nh"], c["hd"])


def _lens(c, g):
    n = torch.randint(c["keys"] // 2 + 1, c["keys"] + 1, (c["batch"],), generator=g, device=DEV)
    n[0] = c["keys"]
    return n.tolist()


# ------------------------------------------------------------------ what a program keeps

def _workspace(a):
    n = ops.attn_workspace_bytes(a)
    ws = torch.empty(max(n, 16), dtype=torch.uint8, device=DEV)
    a.workspace, a.ws_bytes = ws.data_ptr(), n
    return ws


def _prepare_step(c, g):
    cap, start, klen = _step_span(c)
    nh, nkv, hd, s = c["nh"], c["nkv"], c["hd"], c["S"]
    k, v, q = _step_inputs(c, g)
    slots = (torch.arange(start, start + klen - s, device=DEV)) % cap
    kc, ks = _pack(k[: klen - s], c["fmt"], cap, slots)
    vc, vs = _pack(v[: klen - s], c["fmt"], cap, slots)
    st = {"c": c, "kc": kc, "vc": vc, "ks": ks, "vs": vs, "q": q.to(TT[c["io"]]).contiguous(), "nk": k[klen - s:].contiguous(), "nv": v[klen - s:].contiguous(), "cap": cap}
    st["out"] = torch.empty((s, nh, hd), dtype=TT[c["io"]], device=DEV)
    a = ops.make_args(q=st["q"], k_cache=kc, v_cache=vc, k_scales=ks, v_scales=vs, out=st["out"], kv_fmt=FMT[c["fmt"]], q_type=ET[c["io"]], out_type=ET[c["io"]],
                      S=s, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd, cache_hd=hd, cache_cap=cap, win_start=start, klen=klen, window=c["window"],
                      softmax_scale=hd ** -0.5, flags=ops.SETTLED_CACHE)
    if c["append"] == "fused":
        a.new_k, a.new_v, a.n_new, a.new_base_pos = st["nk"].data_ptr(), st["nv"].data_ptr(), s, c["keys"] - s
    st["ws"], st["a"] = _workspace(a), a
    return st


def _run_step(st):
    c = st["c"]
    if c["append"] == "call":
        nkv, hd, s = c["nkv"], c["hd"], c["S"]
        if c["fmt"] == "i8":
            ops.gpu_append_quant_kv_i8(None, st["nk"], st["nv"], st["kc"], st["vc"], st["ks"], st["vs"], s, nkv, hd, nkv * hd, st["cap"], hd, c["keys"] - s)
        else:
            ops.gpu_append_quant_kv_i4(None, st["nk"], st["nv"], st["kc"], st["vc"], st["ks"], st["vs"], s, nkv, hd, nkv * hd, st["cap"], hd, c["keys"] - s,
                                       hd // 32 if c["fmt"] == "i4b32" else 1)
    ops.attn_fused(None, st["a"])
    return {"out": st["out"], "k": st["kc"], "v": st["vc"], "ks": st["ks"], "vs": st["vs"]}


def _exact_step(c, g):
    k, v, q = _step_inputs(c, g)
    q = q.to(TT[c["io"]])
    return {"out": _attend(q, _dequant(k, c["fmt"]), _dequant(v, c["fmt"]), k.shape[0] - c["S"], c["window"], c["hd"] ** -0.5),
            "k": None, "v": None, "ks": None, "vs": None}


def _paged_inputs(c, g):
    lens = _lens(c, g)
    rows = [_rows(g, n, c["nkv"], 128) for n in lens]
    return lens, rows, _normal(g, c["batch"], c["nh"], 128)


def _prepare_paged(c, g):
    lens, rows, q = _paged_inputs(c, g)
    nkv, b = c["nkv"], c["batch"]
    per = (c["keys"] + 127) // 128
    pages = b * per
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32).view(b, per).contiguous()
    kp = torch.zeros((pages, nkv, 128, 128), dtype=torch.int8, device=DEV)
    vp = torch.zeros_like(kp)
    ksp = torch.ones((pages, nkv, 128), device=DEV)
    vsp = torch.ones_like(ksp)
    for i, n in enumerate(lens):
        for x, pool, sp in ((rows[i][0], kp, ksp), (rows[i][1], vp, vsp)):
            plane, buf = _pack(x[: n - 1], "i8", per * 128, torch.arange(n - 1, device=DEV))
            pool[table[i].long()] = plane.view(nkv, per, 128, 128).transpose(0, 1)
            sp[table[i].long()] = buf.view(torch.float32).view(nkv, per, 128).transpose(0, 1)
    st = {"c": c, "kp": kp, "vp": vp, "ksp": ksp, "vsp": vsp, "table": table, "q": q.to(TT[c["io"]]), "per": per, "pages": pages}
    st["nk"] = torch.stack([r[0][-1] for r in rows]).contiguous()
    st["nv"] = torch.stack([r[1][-1] for r in rows]).contiguous()
    st["lens"] = torch.tensor(lens, dtype=torch.int32, device=DEV)
    st["pos"] = st["lens"] - 1
    st["out"] = torch.empty((b, c["nh"], 128), dtype=TT[c["io"]], device=DEV)
    st["wsb"] = ops.attn_paged_workspace_bytes(b, c["nh"], nkv, c["nh"] // nkv, 128, c["keys"])
    st["ws"] = torch.empty(max(st["wsb"], 16), dtype=torch.uint8, device=DEV)
    return st


def _run_paged(st):
    c = st["c"]
    ops.kv_paged_append_quant_i8(None, st["nk"], st["nv"], st["kp"], st["vp"], st["ksp"], st["vsp"], st["table"], st["pos"], batch=c["batch"], nkv=c["nkv"], l_hd=128,
                                 l_kvd=c["nkv"] * 128, max_pages=st["per"])
    ops.attn_paged_decode_i8(None, st["q"], st["kp"], st["vp"], st["ksp"], st["vsp"], st["table"], st["lens"], st["out"], st["ws"], st["wsb"], batch=c["batch"], nh=c["nh"],
                             nkv=c["nkv"], kvg=c["nh"] // c["nkv"], l_hd=128, n_pages=st["pages"], max_pages=st["per"], max_len=c["keys"], softmax_scale=128 ** -0.5,
                             q_type=ET[c["io"]], out_type=ET[c["io"]])
    return {"out": st["out"], "k": st["kp"], "v": st["vp"], "ks": st["ksp"], "vs": st["vsp"]}


def _exact_paged(c, g):
    lens, rows, q = _paged_inputs(c, g)
    q = q.to(TT[c["io"]])
    out = [_attend(q[i][None], _dequant(rows[i][0], "i8"), _dequant(rows[i][1], "i8"), n - 1, 0, 128 ** -0.5)[0] for i, n in enumerate(lens)]
    return {"out": torch.stack(out), "k": None, "v": None, "ks": None, "vs": None}


def _prepare_prompt(c, g):
    nh, nkv, hd, s, t = c["nh"], c["nkv"], c["hd"], c["S"], c["keys"]
    k, v, q = _prompt_inputs(c, g)
    cap = t + 7 & ~7
    slots = torch.arange(t, device=DEV)
    kc, ks = _pack(k, c["fmt"], cap, slots)
    vc, vs = _pack(v, c["fmt"], cap, slots)
    st = {"c": c, "kc": kc, "vc": vc, "ks": ks, "vs": vs, "cap": cap}
    st["out"] = torch.empty((s, nh, hd), dtype=TT[c["io"]] if c["api"] == "fused" else torch.float32, device=DEV)
    if c["api"] == "fused":
        st["q"] = q.to(TT[c["io"]]).contiguous()
        a = ops.make_args(q=st["q"], k_cache=kc, v_cache=vc, k_scales=ks, v_scales=vs, out=st["out"], kv_fmt=FMT[c["fmt"]], q_type=ET[c["io"]], out_type=ET[c["io"]],
                          S=s, nh=nh, nkv=nkv, kvg=nh // nkv, l_hd=hd, cache_hd=hd, cache_cap=cap, klen=t, window=c["window"], softmax_scale=hd ** -0.5)
        st["ws"], st["a"] = _workspace(a), a
    else:
        # the prefix operator applies no softmax scale: the query rows carry it
        st["q"] = (q * hd ** -0.5).contiguous()
        st["scores"] = torch.empty(s * nh * t, device=DEV)
        st["qt"] = torch.empty_like(st["q"])
        st["at"] = torch.empty_like(st["q"])
        if c["fmt"] != "i8":
            st["view"] = [torch.empty((nkv, cap, hd), dtype=torch.int8, device=DEV) for _ in range(2)] + [torch.empty((nkv, cap), device=DEV) for _ in range(2)]
    return st


def _run_prompt(st):
    c = st["c"]
    if c["api"] == "fused":
        ops.attn_fused(None, st["a"])
        return st["out"]
    kc, vc, ks, vs = st["kc"], st["vc"], st["ks"], st["vs"]
    nh, nkv, hd, s, t, cap = c["nh"], c["nkv"], c["hd"], c["S"], c["keys"], st["cap"]
    if c["fmt"] != "i8":
        k8, v8, k8s, v8s = st["view"]
        nb = hd // 32 if c["fmt"] == "i4b32" else 1
        ops.gpu_dequant_kv_i4_to_q8_layer(None, kc, ks, k8, k8s, nkv, t, hd, cap, cap, 0, nb)
        ops.gpu_dequant_kv_i4_to_q8_layer(None, vc, vs, v8, v8s, nkv, t, hd, cap, cap, 0, nb)
        kc, vc, ks, vs = k8, v8, k8s, v8s
    ops.attention_prefill_prefix_batched_int8(None, st["q"], st["qt"], st["scores"], st["at"], st["out"], kc, vc, ks, vs, nh, nkv, hd, hd, cap, s, t, nh // nkv, c["window"], t - s, 0)
    return st["out"]


def _exact_prompt(c, g):
    k, v, q = _prompt_inputs(c, g)
    if c["api"] == "fused":
        return _attend(q.to(TT[c["io"]]), _dequant(k, c["fmt"]), _dequant(v, c["fmt"]), c["keys"] - c["S"], c["window"], c["hd"] ** -0.5)
    seen = _via_q8 if c["fmt"] == "i4b32" else lambda x: _dequant(x, c["fmt"])
    return _attend(q * c["hd"] ** -0.5, seen(k), seen(v), c["keys"] - c["S"], c["window"], 1.0)


def _prepare_rows(c, g):
    nkv, hd, s, cap = c["nkv"], c["hd"], c["S"], c["cap"]
    k, v = _rows(g, s, nkv, hd)
    row = hd if c["fmt"] == "i8" else hd // 2
    st = {"c": c, "k": k, "v": v, "q": _normal(g, s, c["nh"], hd), "qw": 1 + 0.1 * _normal(g, hd), "kw": 1 + 0.1 * _normal(g, hd)}
    st["kc"], st["vc"] = (torch.zeros((nkv, cap, row), dtype=torch.uint8, device=DEV) for _ in range(2))
    st["ks"], st["vs"] = (torch.zeros(_scale_bytes(c["fmt"], nkv, cap, hd), dtype=torch.uint8, device=DEV) for _ in range(2))
    return st


def _run_rows(st):
    c = st["c"]
    ops.kv_norm_rope_append(None, st["q"], st["qw"], st["k"], st["v"], st["kw"], st["kc"], st["vc"], st["ks"], st["vs"], n_s=c["S"], nh=c["nh"], nkv=c["nkv"], l_hd=c["hd"],
                            l_kvd=c["nkv"] * c["hd"], cache_cap=c["cap"], cache_hd=c["hd"], base_pos=c["cap"] - c["S"] // 2, theta=10000.0, rope_dim=c["hd"], kv_fmt=FMT[c["fmt"]])
    return {"q": st["q"], "k": st["kc"], "v": st["vc"], "ks": st["ks"], "vs": st["vs"]}


def _exact_rows(c, g):
    st = _prepare_rows(c, g)
    hd = c["hd"]
    x = st["q"].double()
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * st["qw"].double()
    i = torch.arange(hd // 2, device=DEV, dtype=torch.float64)
    pos = torch.arange(c["S"], device=DEV, dtype=torch.float64)[:, None, None] + (c["cap"] - c["S"] // 2)
    ang = pos * torch.exp(-(2 * i / hd) * math.log(10000.0))
    a, b = x[..., : hd // 2], x[..., hd // 2:]
    q = torch.cat([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1)
    return {"q": q, "k": None, "v": None, "ks": None, "vs": None}


def _dense_inputs(c, g):
    k, v = _rows(g, c["keys"], c["nkv"], c["hd"])
    return k, v, _normal(g, c["S"], c["nh"], c["hd"]) * c["hd"] ** -0.5


def _prepare_dense(c, g):
    k, v, q = _dense_inputs(c, g)
    cap = c["keys"] + 7 & ~7
    st = {"c": c, "q": q, "cap": cap, "out": torch.empty_like(q), "scores": torch.empty(c["S"] * c["nh"] * c["keys"], device=DEV)}
    for n, x in (("kc", k), ("vc", v)):
        st[n] = torch.zeros((c["nkv"], cap, c["hd"]), dtype=TT[c["kv"]], device=DEV)
        st[n][:, : c["keys"]] = x.transpose(0, 1).to(TT[c["kv"]])
    return st


def _run_dense(st):
    c = st["c"]
    nh, nkv, hd, s, t, cap = c["nh"], c["nkv"], c["hd"], c["S"], c["keys"], st["cap"]
    if s == 1 and not c["window"]:
        if c["kv"] == "bf16":
            ops.attention_gpu_bf16_dev(None, None, st["q"], st["kc"], st["vc"], st["scores"], 0, 0, st["out"], nh, nkv, hd, hd, cap, t, nh // nkv)
        else:
            ops.attention_gpu_fp32_dev(None, None, st["q"], st["kc"], st["vc"], st["scores"], st["out"], nh, nkv, hd, hd, cap, t, nh // nkv)
    elif c["kv"] == "bf16":
        ops.attention_prefill_prefix_batched_bf16(None, None, st["q"], 0, 0, st["scores"], 0, 0, st["out"], st["kc"], st["vc"], nh, nkv, hd, hd, cap, s, t, nh // nkv, c["window"], t - s, 0)
    else:
        ops.attention_prefill_prefix_batched_fp32(None, None, st["q"], 0, st["scores"], 0, st["out"], st["kc"], st["vc"], nh, nkv, hd, hd, cap, s, t, nh // nkv, c["window"], t - s, 0)
    return st["out"]


def _exact_dense(c, g):
    k, v, q = _dense_inputs(c, g)
    return _attend(q, k.to(TT[c["kv"]]), v.to(TT[c["kv"]]), c["keys"] - c["S"], c["window"], 1.0)


_PREPARE = {"step": _prepare_step, "paged": _prepare_paged, "prompt": _prepare_prompt, "rows": _prepare_rows, "dense": _prepare_dense}
_RUN = {"step": _run_step, "paged": _run_paged, "prompt": _run_prompt, "rows": _run_rows, "dense": _run_dense}
_EXACT = {"step": _exact_step, "paged": _exact_paged, "prompt": _exact_prompt, "rows": _exact_rows, "dense": _exact_dense}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, _gen(seed))


def run(state):
    return _RUN[state["c"]["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, _gen(seed))


# ------------------------------------------------------------------ what a pass cannot do without

def _pairs(s, t, window):
    """(query row, key) pairs of S rows that are the last of t keys."""
    return sum(min(t - s + r + 1, window) if window else t - s + r + 1 for r in range(s))


def work(case):
    c = case
    nh, nkv, hd, s = c["nh"], c["nkv"], c.get("hd", 128), c.get("S", 1)
    io = 2 if c.get("io") == "bf16" else 4
    if c["kind"] == "paged":
        n = c["batch"] * c["keys"] * 3 // 4                       # lengths are uniform between half of `keys` and all
        return {"bytes": 2 * nkv * n * 132 + c["batch"] * (2 * nh * 128 * io + 2 * nkv * 128 * 4), "flops": 4 * nh * 128 * n}
    if c["kind"] == "rows":
        plane = 2 * s * nkv * (hd if c["fmt"] == "i8" else hd // 2) + 2 * _scale_bytes(c["fmt"], nkv, s, hd)
        return {"bytes": 2 * s * nkv * hd * 4 + 2 * s * nh * hd * 4 + plane, "flops": 0}
    if c["kind"] == "dense":
        keys = min(c["keys"], c["window"] + s - 1) if c["window"] else c["keys"]
        e = 2 if c["kv"] == "bf16" else 4
        return {"bytes": 2 * nkv * keys * hd * e + 2 * s * nh * hd * 4, "flops": 4 * nh * hd * _pairs(s, c["keys"], c["window"])}
    keys = min(c["keys"], c["window"] + s - 1) if c["window"] else c["keys"]
    row = hd if c["fmt"] == "i8" else hd // 2
    by = 2 * nkv * keys * row + 2 * _scale_bytes(c["fmt"], nkv, keys, hd) + 2 * s * nh * hd * io
    if c["kind"] == "step":
        by += 2 * s * nkv * hd * 4
    elif c["api"] == "prefix" and c["fmt"] != "i8":               # the int8 view is written and read again
        by += 2 * 2 * nkv * c["keys"] * (hd + 4)
    return {"bytes": by, "flops": 4 * nh * hd * _pairs(s, c["keys"], c["window"])}


def tolerance(case):
    """About four times the error against exact(): 1.7e-3 for bf16 outputs (their own rounding), 5e-5 for fp32 outputs
    over quantised caches (16-bit fixed-point query limbs), 4e-5 for the rotated rows (fp32 angles at positions of
    thousands), 6e-7 for the dense fp32 sums.  Codes and scale bytes written to a cache stay the same."""
    if case["kind"] == "dense":
        return {"rel": 3e-6, "max": 1e-4}
    if case["kind"] == "rows":
        return {"rel": 2e-4, "max": 4e-3, "differ": 0.0}
    if case["io"] == "bf16" and case.get("api") != "prefix":
        return {"rel": 7e-3, "max": 3e-2, "differ": 0.0}
    return {"rel": 2e-4, "max": 2e-3, "differ": 0.0}
