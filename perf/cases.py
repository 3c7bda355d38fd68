"""The work this library is used for, as cases that can be timed and checked.

A case is a dict of plain values.  ``kind`` names the entry point it goes through:

  prefill    ``fa.prefill`` on device buffers that the caller keeps (f16, bf16, e4m3)
  train      ``torch.ops.fa_b200.prefill`` and its gradient through autograd: one training step's attention
  backward   ``fa.backward`` from a forward's saved output and LSE
  decode     ``fa.decode``: one query row per head against a dense cache
  gqa        ``fa.decode_gqa``: grouped-query attention of the newest token(s) over a serving
             cache ``[B, Skv, Hkv, D]`` or over pages, sequences of their own lengths, 16-bit or e4m3
  chunk      ``torch.ops.fa_b200.decode_gqa``: a chunk of a prompt appended to a cached prefix

``listed`` gives the fixed cases, ``draw`` one more of the same ranges, ``prepare`` the inputs (iid
N(0,1), as everywhere in this repository's tests and benchmark) with the buffers a program keeps,
``run`` one pass, ``exact`` the same in 64 bits without this library.
"""
from __future__ import annotations

import math

import torch

from __graft_entry__ import load_module, load_package

fa = load_package()
load_module("torch_op")

DEV = "cuda"
TYPES = {"f16": torch.float16, "bf16": torch.bfloat16}
PAGE = 16                 # keys per page of the paged caches
PREFILL_STEPS = 5.5e11    # most floating-point operations of a drawn prefill
CACHE_BYTES = 8.5e9       # most cache bytes of a drawn decode


def listed():
    return [
        # One short prompt: the smallest call, where launch and latency count.
        dict(name="prefill_f16_d64_b1h12s512", kind="prefill", dtype="f16", b=1, h=12, s=512, d=64, causal=True),
        # The benchmark's headline: a batch of medium prompts, small heads.
        dict(name="prefill_f16_d64_b8h12s2048", kind="prefill", dtype="f16", b=8, h=12, s=2048, d=64, causal=True),
        # Long context without a mask (an encoder, or a prefix that sees itself): the largest contraction.
        dict(name="prefill_bf16_d128_h32s8192_full", kind="prefill", dtype="bf16", b=1, h=32, s=8192, d=128,
             causal=False),
        # A causal batch of a length that fills no tile.
        dict(name="prefill_bf16_d128_b3h16s2999", kind="prefill", dtype="bf16", b=3, h=16, s=2999, d=128, causal=True),
        # Quantised inputs with a scale per head.
        dict(name="prefill_e4m3_d128_b8h16s4096", kind="prefill", dtype="e4m3", b=8, h=16, s=4096, d=128, causal=True),
        # Attention of a training step, forward and backward, as autograd runs it.
        dict(name="train_f16_d64_b8h12s2048", kind="train", dtype="f16", b=8, h=12, s=2048, d=64, causal=True),
        # Backward alone at the larger head size and a longer sequence.
        dict(name="backward_bf16_d128_b2h16s4096", kind="backward", dtype="bf16", b=2, h=16, s=4096, d=128,
             causal=True),
        # Decode of a large batch over a long dense cache with the benchmark's 16 splits: the largest traffic.
        dict(name="decode_f16_d128_b32h32kv16384", kind="decode", dtype="f16", b=32, h=32, kv=16384, d=128, splits=16),
        # Decode of two short sequences of odd length, split count left to the library.
        dict(name="decode_bf16_d64_b2h12kv1537", kind="decode", dtype="bf16", b=2, h=12, kv=1537, d=64, splits=0),
        # A serving step: a batch of sequences of different lengths over a paged cache.
        dict(name="gqa_bf16_paged_b16kv4096", kind="gqa", dtype="bf16", b=16, hq=32, hkv=8, kv=4096, d=128, tokens=1,
             paged=True, ragged=True),
        # A serving step over a long 8-bit cache.
        dict(name="gqa_e4m3_b32kv16384", kind="gqa", dtype="e4m3", b=32, hq=32, hkv=8, kv=16384, d=128, tokens=1,
             paged=False, ragged=False),
        # The next 512 tokens of a prompt on a prefix of 3584 cached keys (chunked prefill).
        dict(name="chunk_f16_b8kv4096t512", kind="chunk", dtype="f16", b=8, hq=32, hkv=8, kv=4096, d=128, tokens=512,
             paged=False, ragged=False),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "train", "backward", "decode", "gqa", "gqa", "chunk"])
    dtype = rng.choice(["f16", "bf16"])
    d = rng.choice([64, 128])
    if kind in ("prefill", "train", "backward"):
        if kind == "prefill" and rng.random() < 0.3:
            dtype, d = "e4m3", 128
        b, h, s = _log(rng, 1, 8), rng.randint(4, 32), _log(rng, 100, 8192)
        causal = rng.random() < 0.7
        while 4.0 * b * h * s * s * d * (0.5 if causal else 1.0) * (1.0 if kind == "prefill" else 3.5) > PREFILL_STEPS:
            s = s * 3 // 4
        return dict(kind=kind, dtype=dtype, b=b, h=h, s=s, d=d, causal=causal)
    if kind == "decode":
        b, h, kv = _log(rng, 1, 32), rng.randint(4, 32), _log(rng, 200, 32768)
        while 4.0 * b * h * kv * d > CACHE_BYTES:
            kv = kv * 3 // 4
        return dict(kind=kind, dtype=dtype, b=b, h=h, kv=kv, d=d, splits=rng.choice([0, 0, 4, 16]))
    hkv, group = rng.choice([1, 2, 4, 8]), rng.choice([1, 4, 5, 8])
    b, kv = _log(rng, 1, 32), _log(rng, 200, 32768)
    if kind == "gqa":
        if rng.random() < 0.3:
            dtype, d = "e4m3", 128
        while 4.0 * b * hkv * kv * d > CACHE_BYTES:
            kv = kv * 3 // 4
        return dict(kind=kind, dtype=dtype, b=b, hq=hkv * group, hkv=hkv, kv=kv, d=d, tokens=rng.choice([1, 1, 1, 4]),
                    paged=rng.random() < 0.5, ragged=rng.random() < 0.6)
    kv = min(kv, 8192)
    tokens = _log(rng, 64, min(kv, 1024))
    while 4.0 * b * hkv * group * tokens * kv * d > PREFILL_STEPS:
        b = max(1, b * 3 // 4) if b > 1 else 1
        tokens = max(64, tokens * 3 // 4)
    return dict(kind=kind, dtype=dtype, b=b, hq=hkv * group, hkv=hkv, kv=kv, d=d, tokens=tokens, paged=False, ragged=False)


# ------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, dtype, *shape):
    if math.prod(shape) <= 1 << 28:
        return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).to(dtype)
    out = torch.empty(shape, device=DEV, dtype=dtype)            # large caches: piece by piece
    for part in out:
        part.copy_(torch.randn(part.shape, generator=g, device=DEV, dtype=torch.float32))
    return out


def _quantised(g, heads_dim, *shape):
    """e4m3 codes and absmax scales, one for each entry of the first two axes (after moving `heads_dim` to axis 1)."""
    codes = torch.empty(shape, device=DEV, dtype=torch.float8_e4m3fn)
    scales = []
    for part in codes:                                           # per sequence
        x = torch.randn(part.shape, generator=g, device=DEV, dtype=torch.float32)
        axes = [a for a in range(x.dim()) if a != heads_dim - 1]
        sc = x.abs().amax(dim=axes) / 448.0
        view = [1] * x.dim()
        view[heads_dim - 1] = -1
        part.copy_((x / sc.view(view)).to(torch.float8_e4m3fn))
        scales.append(sc)
    return codes, torch.cat(scales).contiguous()


def prepare(case, seed):
    return dict(case=case, **{"prefill": _prepare_dense, "train": _prepare_dense, "backward": _prepare_dense,
                              "decode": _prepare_decode, "gqa": _prepare_cache, "chunk": _prepare_cache}[case["kind"]](case, seed))


def _prepare_dense(c, seed):
    g = _generator(seed)
    shape = (c["b"], c["h"], c["s"], c["d"])
    st = dict(scale=1.0 / math.sqrt(c["d"]))
    if c["dtype"] == "e4m3":
        for n in "qkv":
            st[n], st[n + "_scale"] = _quantised(g, 1, *shape)
        st["o"] = torch.empty(shape, device=DEV, dtype=torch.bfloat16)
    else:
        t = TYPES[c["dtype"]]
        for n in "qkv":
            st[n] = _normal(g, t, *shape).requires_grad_(c["kind"] == "train")
        if c["kind"] != "prefill":
            st["d_o"] = _normal(g, t, *shape)
        st["o"] = torch.empty(shape, device=DEV, dtype=t)
    st["lse"] = torch.empty(shape[:3], device=DEV, dtype=torch.float32)
    if c["kind"] == "backward":                                  # what the forward left behind
        for n in ("dq", "dk", "dv"):
            st[n] = torch.empty_like(st["q"])
        st["ws"] = torch.empty(fa.backward_workspace_bytes(*shape[:3]), device=DEV, dtype=torch.uint8)
        fa.prefill(st["q"], st["k"], st["v"], st["o"], st["lse"], *shape, st["scale"], c["causal"], dtype=c["dtype"],
                   stream=torch.cuda.current_stream())
    return st


def _prepare_decode(c, seed):
    g, t = _generator(seed), TYPES[c["dtype"]]
    b, h, kv, d = c["b"], c["h"], c["kv"], c["d"]
    st = dict(scale=1.0 / math.sqrt(d), q=_normal(g, t, b, h, 1, d), k=_normal(g, t, b, h, kv, d),
              v=_normal(g, t, b, h, kv, d), o=torch.empty((b, h, 1, d), device=DEV, dtype=t),
              lse=torch.empty((b, h, 1), device=DEV, dtype=torch.float32))
    st["splits"] = c["splits"] or fa.decode_default_splits(b, h, kv)
    st["ws_bytes"] = fa.decode_workspace_bytes(b, h, d, st["splits"])
    st["ws"] = torch.empty(st["ws_bytes"], device=DEV, dtype=torch.uint8)
    return st


def _prepare_cache(c, seed):
    g = _generator(seed)
    b, hq, hkv, kv, d, tok = c["b"], c["hq"], c["hkv"], c["kv"], c["d"], c["tokens"]
    st = dict(scale=1.0 / math.sqrt(d))
    n_pages = -(-kv // PAGE)
    rows = n_pages * PAGE if c["paged"] else kv
    if c["dtype"] == "e4m3":
        # the query heads of a group share the scale of their KV head
        q, qs = _quantised(g, 1, b, hkv, tok, hq // hkv, d)
        st["q"], st["q_scale"] = q.permute(0, 2, 1, 3, 4).reshape(b, tok, hq, d).contiguous(), qs
        for n in "kv":
            st[n], st[n + "_scale"] = _quantised(g, 2, b, rows, hkv, d)
        out = torch.bfloat16
    else:
        out = TYPES[c["dtype"]]
        st["q"] = _normal(g, out, b, tok, hq, d)
        for n in "kv":
            st[n] = _normal(g, out, b, rows, hkv, d)
    if c["ragged"]:
        lens = torch.randint(min(kv, max(tok, kv // 16)), kv + 1, (b,), generator=g, device=DEV, dtype=torch.int32)
        lens[0] = kv
        st["lens"] = lens
    if c["paged"]:                                               # the sequences' pages lie shuffled in one pool
        st["table"] = torch.randperm(b * n_pages, generator=g, device=DEV).to(torch.int32).view(b, n_pages)
        for n in "kv":
            pool = torch.empty_like(st[n]).view(torch.uint8).view(b * n_pages, -1)
            pool[st["table"].flatten().long()] = st[n].view(torch.uint8).view(b * n_pages, -1)
            st[n] = pool.view(st[n].dtype).view(b * n_pages, PAGE, hkv, d)
    if c["kind"] == "gqa":
        st["o"] = torch.empty((b, tok, hq, d), device=DEV, dtype=out)
        st["lse"] = torch.empty((b, tok, hq), device=DEV, dtype=torch.float32)
        kw = dict(dtype=c["dtype"], num_q_tokens=tok)
        if c["paged"]:
            kw.update(kv_strides=(0, d, hkv * d), block_table=st["table"], block_table_stride=n_pages, page_size=PAGE,
                      num_pages=b * n_pages, kv_page_stride=PAGE * hkv * d)
        else:
            kw.update(kv_strides=(kv * hkv * d, d, hkv * d))
        if c["ragged"]:
            kw.update(seq_lens=st["lens"])
        if c["dtype"] == "e4m3":
            kw.update(q_scale=st["q_scale"], k_scale=st["k_scale"], v_scale=st["v_scale"])
        per_tile = max(1, min(tok, 128 // (hq // hkv)))
        splits = fa.decode_gqa_default_splits(b * -(-tok // per_tile), hkv, kv)
        st["ws_bytes"] = fa.decode_workspace_bytes(b, tok * hq, d, splits)
        st["ws"] = torch.empty(st["ws_bytes"], device=DEV, dtype=torch.uint8)
        st["kw"] = kw
    return st


# ------------------------------------------------------------------------------------------- one pass
def run(state):
    c, st = state["case"], state
    stream = torch.cuda.current_stream()
    if c["kind"] == "prefill":
        kw = dict(dtype=c["dtype"], stream=stream)
        if c["dtype"] == "e4m3":
            kw.update(q_scale=st["q_scale"], k_scale=st["k_scale"], v_scale=st["v_scale"])
        fa.prefill(st["q"], st["k"], st["v"], st["o"], st["lse"], c["b"], c["h"], c["s"], c["d"], st["scale"], c["causal"], **kw)
        return st["o"], st["lse"]
    if c["kind"] == "train":
        o, lse = torch.ops.fa_b200.prefill(st["q"], st["k"], st["v"], st["scale"], c["causal"])
        dq, dk, dv = torch.autograd.grad(o, (st["q"], st["k"], st["v"]), st["d_o"])
        return o.detach(), lse.detach(), dq, dk, dv
    if c["kind"] == "backward":
        fa.backward(st["q"], st["k"], st["v"], st["o"], st["d_o"], st["lse"], st["dq"], st["dk"], st["dv"], c["b"], c["h"],
                    c["s"], c["d"], st["scale"], c["causal"], dtype=c["dtype"], workspace=st["ws"],
                    workspace_bytes=st["ws"].numel(), stream=stream)
        return st["dq"], st["dk"], st["dv"]
    if c["kind"] == "decode":
        fa.decode(st["q"], st["k"], st["v"], st["o"], st["lse"], None, c["b"], c["h"], c["kv"], c["d"], st["scale"],
                  dtype=c["dtype"], num_splits=st["splits"], workspace=st["ws"], workspace_bytes=st["ws_bytes"], stream=stream)
        return st["o"], st["lse"]
    if c["kind"] == "gqa":
        fa.decode_gqa(st["q"], st["k"], st["v"], st["o"], st["lse"], c["b"], c["hq"], c["hkv"], c["kv"], c["d"], st["scale"],
                      workspace=st["ws"], workspace_bytes=st["ws_bytes"], stream=stream, **st["kw"])
        return st["o"], st["lse"]
    return torch.ops.fa_b200.decode_gqa(st["q"], st["k"], st["v"], st["scale"])


# ------------------------------------------------------------------------------------------- what a pass needs
def work(case):
    c = case
    es = 1 if c["dtype"] == "e4m3" else 2
    if c["kind"] in ("prefill", "train", "backward"):
        rows, d, s = c["b"] * c["h"] * c["s"], c["d"], c["s"]
        forward = 4.0 * d * rows * ((s + 1) / 2 if c["causal"] else s)
        tensor = rows * d
        if c["kind"] == "prefill":
            return {"bytes": 3 * tensor * es + 2 * tensor + 4 * rows, "flops": forward}
        if c["kind"] == "train":                                 # in: q k v dO; out: o lse dq dk dv
            return {"bytes": 8 * tensor * es + 4 * rows, "flops": 3.5 * forward}
        return {"bytes": 8 * tensor * es + 4 * rows, "flops": 2.5 * forward}
    if c["kind"] == "decode":
        rows, d, kv = c["b"] * c["h"], c["d"], c["kv"]
        return {"bytes": rows * (2 * kv * d * es + 2 * d * es + 4), "flops": 4.0 * rows * kv * d}
    rows, d, tok = c["b"] * c["tokens"] * c["hq"], c["d"], c["tokens"]
    # ragged lengths are uniform between 1/16 of the maximum and the maximum
    mean = c["kv"] * (17 / 32) if c["ragged"] else float(c["kv"])
    return {"bytes": c["b"] * c["hkv"] * 2 * mean * d * es + rows * d * (es + 2) + 4 * rows,
            "flops": 4.0 * rows * d * max(1.0, mean - (tok - 1) / 2)}


def tolerance(case):
    # Outputs are rounded to 16 bits, and so are the probabilities (and, backward, dS) before they enter
    # the second product; the sums are 32-bit.  Four times what was measured against `exact` over the
    # listed cases and some drawn ones: f16 rel 3.2e-4, max 3.1e-3 forward and 1.5e-2 backward; bf16 (and
    # e4m3 inputs, whose output is bf16) rel 2.5e-3, max 3.0e-2 forward and 1.6e-1 backward (the first rows
    # under the causal mask have gradients far above the mean and dS is rounded relative to them).
    backward = case["kind"] in ("train", "backward")
    if case["dtype"] == "f16":
        return {"rel": 1.3e-3, "max": 6e-2 if backward else 1.3e-2}
    return {"rel": 1e-2, "max": 6.5e-1 if backward else 1.2e-1}


# ------------------------------------------------------------------------------------------- 64 bits
def _attention64(q, k, v, scale, limit):
    """Rows of q [n, m, d] against k, v [n, r, d]; row i sees the first limit[..., i] keys."""
    s = torch.matmul(q, k.transpose(-1, -2)) * scale
    if limit is not None:
        s.masked_fill_(torch.arange(k.shape[-2], device=DEV) >= limit.unsqueeze(-1), -math.inf)
    lse = torch.logsumexp(s, -1)
    s.sub_(lse.unsqueeze(-1)).exp_()
    return torch.matmul(s, v), lse, s


def exact(case, seed):
    c, st = case, prepare(case, seed)
    with torch.no_grad():
        if c["kind"] in ("prefill", "train", "backward"):
            return _exact_dense(c, st)
        if c["kind"] == "decode":
            o, lse = [], []
            for i in range(c["b"]):
                r = _attention64(st["q"][i].double(), st["k"][i].double(), st["v"][i].double(), st["scale"], None)
                o.append(r[0])
                lse.append(r[1])
            return torch.stack(o), torch.stack(lse)
        return _exact_cache(c, st)


def _exact_dense(c, st):
    n, s = c["b"] * c["h"], c["s"]
    limit = torch.arange(1, s + 1, device=DEV) if c["causal"] else None

    def head(name, i):
        x = st[name].detach().reshape(n, s, c["d"])[i].double()
        return x * st[name + "_scale"][i].double() if c["dtype"] == "e4m3" else x

    outs = []
    for i in range(n):
        q, k, v = (head(x, i) for x in "qkv")
        o, lse, p = _attention64(q, k, v, st["scale"], limit)
        if c["kind"] == "prefill":
            outs.append((o, lse))
            continue
        do = head("d_o", i)
        dv = p.T @ do
        ds = p * (do @ v.T - (do * o).sum(-1, keepdim=True)) * st["scale"]
        grads = (ds @ k, ds.T @ q, dv)
        outs.append((o, lse) + grads if c["kind"] == "train" else grads)
    return tuple(torch.stack(x).reshape(c["b"], c["h"], *x[0].shape) for x in zip(*outs))


def _exact_cache(c, st):
    b, hq, hkv, kv, d, tok = c["b"], c["hq"], c["hkv"], c["kv"], c["d"], c["tokens"]
    group = hq // hkv
    o = torch.empty((b, tok, hq, d), device=DEV, dtype=torch.float64)
    lse = torch.empty((b, tok, hq), device=DEV, dtype=torch.float64)
    for i in range(b):
        n = int(st["lens"][i]) if c["ragged"] else kv
        cache = [st[x][st["table"][i].long()].reshape(-1, hkv, d) if c["paged"] else st[x][i] for x in "kv"]
        k, v = (x[:n].double().permute(1, 0, 2) for x in cache)                       # [hkv, n, d]
        q = st["q"][i].double().view(tok, hkv, group, d).permute(1, 0, 2, 3).reshape(hkv, tok * group, d)
        if c["dtype"] == "e4m3":
            q, k, v = (x * st[y + "_scale"].view(b, hkv)[i].double().view(hkv, 1, 1) for x, y in ((q, "q"), (k, "k"), (v, "v")))
        limit = (n - tok + 1 + torch.arange(tok, device=DEV)).repeat_interleave(group)
        for h in range(hkv):
            oh, lh, _ = _attention64(q[h], k[h], v[h], st["scale"], limit)
            o[i, :, h * group:(h + 1) * group] = oh.view(tok, group, d)
            lse[i, :, h * group:(h + 1) * group] = lh.view(tok, group)
    return o, lse
