"""Decode whose query tile has few live rows: up to 8, up to 16 (the 16-lane TMEM shapes) and just above, with
score maxima that rise from key tile to key tile so that O is rescaled, ragged lengths and several KV splits.
Against the CPU oracle; fp16 O 2e-3, LSE 1e-3 (max abs), e4m3 O 3e-2."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def check_rows(fa, oracle, o, lse, q, k, v, lens, scale, tol):
    b, t, hq, d = q.shape
    group = hq // k.shape[2]
    for i in range(b):
        n = int(lens[i])
        for h in range(hq):
            for tok in range(t):
                vis = n - t + tok + 1
                got = o[i, tok, h].float().cpu().numpy()
                if vis <= 0:
                    assert (got == 0).all() and float(lse[i, tok, h]) == -np.inf
                    continue
                kk, vv = (x[i, :vis, h // group].cpu().numpy()[None] for x in (k, v))
                ref, l_ref = oracle.attention(q[i, tok, h].cpu().numpy()[None, None], kk, vv, scale, False)
                assert np.abs(got - ref[0, 0]).max() < tol and abs(float(lse[i, tok, h]) - l_ref[0, 0]) < 1e-3, (i, h, tok)


@pytest.mark.parametrize("group,t", [(1, 1), (3, 1), (8, 1), (9, 1), (4, 3), (16, 1), (8, 2), (17, 1), (6, 3)])
@pytest.mark.parametrize("d,splits,rising", [(128, 1, False), (128, 3, True), (64, 2, True)])
def test_few_live_rows(fa, oracle, dev, group, t, d, splits, rising):
    b, hkv, skv = 3, 2, 900
    gen = torch.Generator(device=dev).manual_seed(group * 100 + t)
    q = torch.randn((b, t, group * hkv, d), generator=gen, device=dev).half()
    k, v = (torch.randn((b, skv, hkv, d), generator=gen, device=dev).half() for _ in range(2))
    if rising:
        q[..., 0] = 4.0
        k[..., 0] = ((torch.arange(skv, device=dev) // 128) * 24.0).half()[None, :, None]
    lens = torch.tensor([skv, 1, 515], device=dev, dtype=torch.int32)
    scale = 0.125
    o = torch.full_like(q, float("nan"))
    lse = torch.full((b, t, group * hkv), float("nan"), device=dev)
    wsb = fa.decode_workspace_bytes(b, t * group * hkv, d, splits)
    ws = torch.empty(wsb, device=dev, dtype=torch.uint8)
    fa.decode_gqa(q, k, v, o, lse, b, group * hkv, hkv, skv, d, scale, num_splits=splits, kv_strides=(skv * hkv * d, d, hkv * d),
                  num_q_tokens=t, seq_lens=lens, workspace=ws, workspace_bytes=wsb)
    torch.cuda.synchronize()
    assert fa.device_status() == 0
    check_rows(fa, oracle, o, lse, q.float(), k.float(), v.float(), lens.cpu(), scale, 2e-3)


@pytest.mark.parametrize("group,t,skv", [(4, 1, 130), (4, 1, 1700), (8, 2, 700), (12, 1, 700), (20, 1, 700)])
def test_e4m3_stages(fa, oracle, dev, group, t, skv):
    """From fewer key tiles than load stages to several times as many."""
    b, hkv, d = 2, 2, 128
    gen = torch.Generator(device=dev).manual_seed(skv + group)
    qf, kf, vf = (torch.randn(s, generator=gen, device=dev) for s in ((b, t, group * hkv, d), (b, skv, hkv, d), (b, skv, hkv, d)))
    q, k, v = (x.to(torch.float8_e4m3fn) for x in (qf, kf, vf))
    sc = torch.ones((3, b * hkv), device=dev)
    lens = torch.tensor([skv, skv - 129], device=dev, dtype=torch.int32)
    o = torch.full((b, t, group * hkv, d), float("nan"), device=dev, dtype=torch.bfloat16)
    lse = torch.full((b, t, group * hkv), float("nan"), device=dev)
    wsb = fa.decode_workspace_bytes(b, t * group * hkv, d, 2)
    ws = torch.empty(wsb, device=dev, dtype=torch.uint8)
    fa.decode_gqa(q, k, v, o, lse, b, group * hkv, hkv, skv, d, 0.1, dtype="e4m3", num_splits=2, kv_strides=(skv * hkv * d, d, hkv * d),
                  num_q_tokens=t, seq_lens=lens, q_scale=sc[0], k_scale=sc[1], v_scale=sc[2], workspace=ws, workspace_bytes=wsb)
    torch.cuda.synchronize()
    assert fa.device_status() == 0
    check_rows(fa, oracle, o, lse, q.float(), k.float(), v.float(), lens.cpu(), 0.1, 3e-2)
