"""Chunks of new tokens over a cache (``fa_decode_gqa`` with num_q_tokens > 1): query tiles that their
group does not fill, the last tile of a chunk, and caches larger than L2, whose heads are walked a few at
a time.  Against the CPU oracle; tolerances of the path: fp16 O 2e-3, e4m3 inputs 3e-2, LSE 1e-3 (max abs)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def run_chunk(fa, dev, q, k, v, scale, seq_lens=None, splits=1):
    b, t, hq, d = q.shape
    skv, hkv = k.shape[1], k.shape[2]
    o = torch.full_like(q, float("nan"))
    lse = torch.full((b, t, hq), float("nan"), device=dev, dtype=torch.float32)
    wsb = fa.decode_workspace_bytes(b, t * hq, d, splits)
    ws = torch.empty(wsb, device=dev, dtype=torch.uint8)
    fa.decode_gqa(q, k, v, o, lse, b, hq, hkv, skv, d, scale, num_splits=splits, kv_strides=(skv * hkv * d, d, hkv * d),
                  num_q_tokens=t, workspace=ws, workspace_bytes=wsb, seq_lens=seq_lens)
    torch.cuda.synchronize()
    assert fa.device_status() == 0
    return o, lse


def check(oracle, q, k, v, o, lse, scale, n, b, heads, tokens, tol=2e-3):
    """Oracle on the given query heads and tokens of sequence b, whose cache holds n keys."""
    t, hq = q.shape[1], q.shape[2]
    group = hq // k.shape[2]
    for h in heads:
        kh, vh = (x[b, :n, h // group].float().cpu().numpy()[None] for x in (k, v))
        for i in tokens:
            vis = n - t + i + 1
            got_o, got_l = o[b, i, h].float().cpu().numpy(), float(lse[b, i, h])
            if vis <= 0:
                assert (got_o == 0).all() and got_l == -np.inf
                continue
            o_ref, l_ref = oracle.attention(q[b, i, h].float().cpu().numpy()[None, None], kh[:, :vis], vh[:, :vis], scale, False)
            assert np.abs(got_o - o_ref[0, 0]).max() < tol and abs(got_l - l_ref[0, 0]) < 1e-3, (b, h, i)


@pytest.mark.parametrize("group,t", [(1, 33), (1, 200), (3, 43), (5, 60), (7, 19), (32, 9), (128, 2)])
@pytest.mark.parametrize("d", [64, 128])
def test_partly_filled_query_tiles(fa, dev, oracle, group, t, d):
    """live rows from 33 to 128, chunks that end inside a tile, one sequence shorter than the chunk."""
    b, hkv, skv = 3, 2, 300
    gen = torch.Generator(device=dev).manual_seed(group * 1000 + t)
    q = torch.randn((b, t, group * hkv, d), generator=gen, device=dev).half()
    k, v = (torch.randn((b, skv, hkv, d), generator=gen, device=dev).half() for _ in range(2))
    lens = torch.tensor([skv, max(1, t // 2), 129 if t < 129 else 260], device=dev, dtype=torch.int32)
    scale = float(d) ** -0.5
    o, lse = run_chunk(fa, dev, q, k, v, scale, seq_lens=lens)
    heads = sorted({0, group - 1, group, 2 * group - 1})
    tokens = sorted({0, 1, t // 2, t - 2, t - 1} & set(range(t)))
    for i in range(b):
        check(oracle, q, k, v, o, lse, scale, int(lens[i]), i, heads, tokens)


def test_cache_larger_than_l2(fa, dev, oracle):
    """35 (sequence, KV head) pairs of 2 MB, walked 8 at a time (the last walk has 3, odd walks run light to
    heavy): every pair must match a call of its own bit for bit, some of them the oracle."""
    b, hkv, group, t, skv, d = 5, 7, 2, 150, 4096, 128
    gen = torch.Generator(device=dev).manual_seed(5)
    q = torch.randn((b, t, group * hkv, d), generator=gen, device=dev).half()
    k, v = (torch.randn((b, skv, hkv, d), generator=gen, device=dev).half() for _ in range(2))
    scale = float(d) ** -0.5
    o, lse = run_chunk(fa, dev, q, k, v, scale)
    for i in range(b):
        for h in range(hkv):
            hs = slice(h * group, (h + 1) * group)
            o1, l1 = run_chunk(fa, dev, *(x.contiguous() for x in (q[i:i + 1, :, hs], k[i:i + 1, :, h:h + 1], v[i:i + 1, :, h:h + 1])), scale)
            assert torch.equal(o1[0], o[i, :, hs]) and torch.equal(l1[0], lse[i, :, hs]), (i, h)
    check(oracle, q, k, v, o, lse, scale, skv, 0, [0, 13], [0, 63, 64, 149])
    check(oracle, q, k, v, o, lse, scale, skv, 4, [12, 13], [127, 128, 149])


@pytest.mark.parametrize("group,t", [(1, 33), (3, 43), (4, 70), (5, 60), (128, 2)])
def test_e4m3_partly_filled_query_tiles(fa, dev, oracle, group, t):
    """The same over an e4m3 cache, whose bf16 output leaves through a tensor map of its own: one KV split, live rows
    from 33 to 128, scales per (sequence, KV head), one sequence shorter than the chunk."""
    b, hkv, skv, d = 3, 2, 300, 128
    hq = group * hkv
    gen = torch.Generator(device=dev).manual_seed(group * 1000 + t)
    q, k, v = ((torch.randn(shape, generator=gen, device=dev) * 16).to(torch.float8_e4m3fn)
               for shape in ((b, t, hq, d), (b, skv, hkv, d), (b, skv, hkv, d)))
    qs, ks, vs = ((torch.rand((b, hkv), generator=gen, device=dev) + 0.5) / 16 for _ in range(3))
    lens = torch.tensor([skv, max(1, t // 2), 129 if t < 129 else 260], device=dev, dtype=torch.int32)
    o = torch.full((b, t, hq, d), float("nan"), device=dev, dtype=torch.bfloat16)
    lse = torch.full((b, t, hq), float("nan"), device=dev)
    wsb = fa.decode_workspace_bytes(b, t * hq, d, 1)
    ws = torch.empty(wsb, device=dev, dtype=torch.uint8)
    scale = float(d) ** -0.5
    fa.decode_gqa(q, k, v, o, lse, b, hq, hkv, skv, d, scale, dtype="e4m3", num_splits=1, kv_strides=(skv * hkv * d, d, hkv * d),
                  num_q_tokens=t, workspace=ws, workspace_bytes=wsb, seq_lens=lens, q_scale=qs, k_scale=ks, v_scale=vs)
    torch.cuda.synchronize()
    assert fa.device_status() == 0
    qf = q.float() * qs.repeat_interleave(group, 1)[:, None, :, None]
    kf, vf = (x.float() * sc[:, None, :, None] for x, sc in ((k, ks), (v, vs)))
    heads = sorted({0, group - 1, group, 2 * group - 1})
    tokens = sorted({0, 1, t // 2, t - 2, t - 1} & set(range(t)))
    for i in range(b):
        check(oracle, qf, kf, vf, o, lse, scale, int(lens[i]), i, heads, tokens, tol=3e-2)
