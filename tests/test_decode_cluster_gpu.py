"""Decode in one launch (the CTAs of a head as a cluster) on both sides of its dispatch line, and the merge
kernel with few and many parts.  Tolerances of the decode path: fp16 O 2e-3, LSE 1e-3 (max abs)."""
import numpy as np
import pytest
import torch

from helpers import to_dev

pytestmark = pytest.mark.gpu


def run_decode(fa, dev, q, k, v, scale, dtype, splits):
    bh, kv, d = k.shape
    dq, dk, dv = (to_dev(x, dtype, dev) for x in (q, k, v))
    o = torch.full((bh, d), float("nan"), device=dev, dtype=dq.dtype)
    of = torch.full((bh, d), float("nan"), device=dev, dtype=torch.float32)
    lse = torch.full((bh,), float("nan"), device=dev, dtype=torch.float32)
    n = splits or fa.decode_default_splits(1, bh, kv)
    wsb = fa.decode_workspace_bytes(1, bh, d, n)
    ws = torch.empty(wsb, device=dev, dtype=torch.uint8)
    fa.decode(dq, dk, dv, o, lse, of, 1, bh, kv, d, scale, dtype=dtype, num_splits=splits, workspace=ws, workspace_bytes=wsb)
    torch.cuda.synchronize()
    return o.float().cpu().numpy(), of.cpu().numpy(), lse.cpu().numpy()


@pytest.mark.parametrize("bh,kv,splits", [
    (1, 1, 0), (1, 63, 0), (1, 65, 0), (1, 129, 0), (2, 449, 0),     # clusters of 1 to 8, slices of at least 64 keys
    (24, 1537, 0), (37, 1100, 8), (37, 1100, 1),                     # 8 warps a CTA and 16
    (74, 700, 8), (75, 700, 8),                                      # 592 CTAs: one launch; 600: two
    (148, 300, 2), (600, 140, 1), (5, 10, 4), (3, 2000, 9),
])
@pytest.mark.parametrize("d,dtype", [(64, "bf16"), (128, "f16")])
def test_decode_shapes(fa, dev, oracle, bh, kv, splits, d, dtype):
    q = oracle.round_to(oracle.normal_inputs(bh + kv, (bh, 1, d), n=1)[0], dtype)
    k, v = (oracle.round_to(x, dtype) for x in oracle.normal_inputs(bh * kv, (bh, kv, d), n=2))
    scale = float(d) ** -0.5
    o, of, lse = run_decode(fa, dev, q, k, v, scale, dtype, splits)
    o_ref, l_ref = oracle.attention(q, k, v, scale, False)
    assert np.abs(of - o_ref[:, 0]).max() < 2e-4                     # fp32 sums, before the output is rounded
    # rounding to 16 bits: half an ulp, |O| < 4
    assert np.abs(o - o_ref[:, 0]).max() < (1e-2 if dtype == "bf16" else 2e-3)
    assert np.abs(lse - l_ref[:, 0]).max() < 1e-3


@pytest.mark.parametrize("n_parts", [1, 2, 3, 15, 16, 17, 33, 256])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("packed", [False, True])
def test_combine_part_counts(fa, dev, n_parts, d, packed):
    check_combine(fa, dev, n_parts, 7, d, packed)


@pytest.mark.parametrize("n_parts,rows_per_sm", [(8, 3), (8, 7), (9, 7), (64, 7)])
@pytest.mark.parametrize("beyond", [0, 1])
@pytest.mark.parametrize("d,packed", [(64, True), (128, False)])
def test_combine_row_counts(fa, dev, n_parts, rows_per_sm, beyond, d, packed):
    """Both merge kernels on both sides of the line between them."""
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    check_combine(fa, dev, n_parts, rows_per_sm * sms + beyond, d, packed)


def check_combine(fa, dev, n_parts, rows, d, packed):
    gen = torch.Generator(device=dev).manual_seed(n_parts * d)
    o = torch.randn((n_parts, rows, d), generator=gen, device=dev)
    lse = torch.randn((n_parts, rows), generator=gen, device=dev) * 4
    lse[:, 3] = -float("inf")                                        # a row without keys
    lse[n_parts // 2, 4] = -float("inf")                             # a part without keys
    out = torch.full((rows, d), float("nan"), device=dev, dtype=torch.float16)
    out_l = torch.full((rows,), float("nan"), device=dev)
    if packed:
        fa.combine_packed(torch.cat([o, lse.unsqueeze(-1)], -1).contiguous(), n_parts, rows, d, out, out_l)
    else:
        fa.combine(o, lse, n_parts, rows, d, out, out_l)
    ref_l = torch.logsumexp(lse.double(), 0)
    w = torch.exp(lse.double() - ref_l).nan_to_num(0.0)
    ref = (w.unsqueeze(-1) * o.double()).sum(0)
    assert (out.double() - ref).abs().max() < 2e-3                   # half an fp16 ulp for |O| < 4
    keep = torch.isfinite(ref_l)
    assert (out_l.double() - ref_l)[keep].abs().max() < 1e-4
    assert (out_l[~keep] == -float("inf")).all()
