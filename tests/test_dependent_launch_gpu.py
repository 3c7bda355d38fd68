"""Every kernel starts while the one before it on the stream drains (programmatic dependent launch), so
inputs written by the very previous kernel must be complete when they are read, and buffers that a later
kernel overwrites must have been read.  Each sequence is compared bit for bit with the same calls
separated by synchronisations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rnd(gen, dev, *shape, dtype=torch.float16):
    return torch.randn(shape, generator=gen, device=dev).to(dtype)


def sequence(fa, dev, seed, sync):
    """Calls in a row, every one on data the kernel before it wrote; `sync` between them or nothing."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    b, h, s, d = 2, 40, 700, 64
    src = [rnd(gen, dev, b, h, s, d) for _ in range(4)]
    q, k, v, d_o, o, o2, dq, dk, dv = (torch.zeros_like(src[0]) for _ in range(9))
    lse = torch.zeros((b, h, s), device=dev)
    ws = torch.empty(fa.backward_workspace_bytes(b, h, s), device=dev, dtype=torch.uint8)
    cache = [rnd(gen, dev, 60, 16, 8, 128) for _ in range(2)]               # pages of 16 keys
    kc, vc = (torch.zeros_like(x) for x in cache)
    qd, od, ld = rnd(gen, dev, 4, 32, 128), torch.zeros((4, 32, 128), device=dev, dtype=torch.float16), torch.zeros((4, 32), device=dev)
    table_src = torch.randperm(60, generator=gen, device=dev).to(torch.int32).view(4, 15)
    lens_src = torch.tensor([240, 17, 129, 200], device=dev, dtype=torch.int32)
    table, lens = torch.zeros_like(table_src), torch.zeros_like(lens_src)
    splits = 2
    wsd = torch.empty(fa.decode_workspace_bytes(4, 32, 128, splits), device=dev, dtype=torch.uint8)
    kd, vd = (torch.zeros((8, 1500, 64), device=dev, dtype=torch.float16) for _ in range(2))
    dsrc = [rnd(gen, dev, 8, 1500, 64) for _ in range(2)]
    qs = rnd(gen, dev, 8, 64)
    os_, ls = torch.zeros((8, 64), device=dev, dtype=torch.float16), torch.zeros(8, device=dev)
    ws2 = torch.empty(fa.decode_workspace_bytes(1, 8, 64, 16), device=dev, dtype=torch.uint8)
    q8, k8, v8 = ((x[0, :, :, :].repeat(1, 1, 2) * 16).to(torch.float8_e4m3fn) for x in src[:3])
    scale_src = torch.rand((3, h), generator=gen, device=dev) + 0.5
    scales = torch.zeros_like(scale_src)
    o8 = torch.zeros((h, s, 128), device=dev, dtype=torch.bfloat16)
    stream = torch.cuda.current_stream(dev)
    torch.cuda.synchronize()

    def step(f):
        f()
        if sync:
            torch.cuda.synchronize()

    for x, y in zip((q, k, v, d_o), src):
        step(lambda: x.copy_(y))
    step(lambda: fa.prefill(q, k, v, o, lse, b, h, s, d, 0.125, True, stream=stream))
    step(lambda: fa.backward(q, k, v, o, d_o, lse, dq, dk, dv, b, h, s, d, 0.125, True, workspace=ws, workspace_bytes=ws.numel(), stream=stream))
    step(lambda: fa.prefill(o, dq, dk, o2, None, b, h, s, d, 0.125, False, stream=stream))   # on outputs of both
    step(lambda: dq.mul_(2))                                                 # overwrites what it reads
    step(lambda: kc.copy_(cache[0]))
    step(lambda: vc.copy_(cache[1]))
    step(lambda: table.copy_(table_src))
    step(lambda: lens.copy_(lens_src))
    step(lambda: fa.decode_gqa(qd, kc, vc, od, ld, 4, 32, 8, 240, 128, 0.1, num_splits=splits, kv_strides=(0, 128, 1024), block_table=table,
                               block_table_stride=15, page_size=16, num_pages=60, kv_page_stride=16 * 1024, seq_lens=lens,
                               workspace=wsd, workspace_bytes=wsd.numel(), stream=stream))
    step(lambda: kc.zero_())
    outs = []
    for n in (3, 16):                                                       # one launch, two launches
        step(lambda: kd.copy_(dsrc[0]))
        step(lambda: vd.copy_(dsrc[1]))
        step(lambda: fa.decode(qs, kd, vd, os_, ls, None, 1, 8, 1500, 64, 0.125, num_splits=n, workspace=ws2, workspace_bytes=ws2.numel(), stream=stream))
        step(lambda: kd.zero_())
        outs += [os_.clone(), ls.clone()]
    step(lambda: scales.copy_(scale_src))
    step(lambda: fa.prefill(q8, k8, v8, o8, None, 1, h, s, 128, 0.01, True, dtype="e4m3", q_scale=scales[0], k_scale=scales[1], v_scale=scales[2], stream=stream))
    step(lambda: scales.zero_())
    torch.cuda.synchronize()
    assert fa.device_status() == 0
    return outs + [o, lse, dq, dk, dv, o2, od, ld, o8]


def test_back_to_back_equals_synchronised(fa, dev):
    ref = sequence(fa, dev, 1, True)
    assert all(torch.isfinite(x.float()).all() for x in ref)
    for _ in range(10):
        for x, y in zip(sequence(fa, dev, 1, False), ref):
            assert torch.equal(x, y)


def test_captured_after_a_copy_and_a_join(fa, dev):
    """In a captured graph, behind a copy, a memset and a join with a second stream."""
    gen = torch.Generator(device=dev).manual_seed(2)
    b, h, s, d = 1, 24, 500, 64
    src = [rnd(gen, dev, b, h, s, d) for _ in range(3)]
    q, k, v, o = (torch.zeros_like(src[0]) for _ in range(4))
    host = torch.zeros((b, h, s, d), dtype=torch.float16).pin_memory()
    lse = torch.zeros((b, h, s), device=dev)
    main, side = torch.cuda.Stream(dev), torch.cuda.Stream(dev)

    def enqueue(stream, other):
        q.copy_(src[0])
        other.wait_stream(stream)
        with torch.cuda.stream(other):
            k.copy_(src[1])
            v.copy_(host, non_blocking=True)
        o.zero_()
        stream.wait_stream(other)
        fa.prefill(q, k, v, o, lse, b, h, s, d, 0.125, True, stream=stream)
        fa.prefill(o, k, v, q, None, b, h, s, d, 0.125, True, stream=stream)

    host.copy_(src[2])
    with torch.cuda.stream(main):
        enqueue(main, side)
    torch.cuda.synchronize()
    ref = [q.clone(), lse.clone()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=main):
        enqueue(main, side)
    for _ in range(5):
        q.zero_(), lse.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(q, ref[0]) and torch.equal(lse, ref[1])
    assert fa.device_status() == 0


@pytest.mark.parametrize("d,dtype", [(64, "f16"), (128, "bf16")])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("b,h,s", [(1, 3, 130), (2, 40, 300), (1, 5, 1100)])
def test_backward_calls_in_a_row(fa, dev, d, dtype, causal, b, h, s):
    """Calls on changing data with one workspace: the dQ kernel starts before the dK/dV kernel has ended and reads
    the delta that this call's first kernel has just written over the last call's."""
    gen = torch.Generator(device=dev).manual_seed(s + d)
    t = torch.float16 if dtype == "f16" else torch.bfloat16
    scale = d ** -0.5
    sets = []
    for i in range(3):
        q, k, v, d_o = (rnd(gen, dev, b, h, s, d, dtype=t) * (1 + i) for _ in range(4))
        o, lse = torch.empty_like(q), torch.empty((b, h, s), device=dev)
        fa.prefill(q, k, v, o, lse, b, h, s, d, scale, causal, dtype=dtype)
        sets.append((q, k, v, o, d_o, lse))
    ws = torch.zeros(fa.backward_workspace_bytes(b, h, s), device=dev, dtype=torch.uint8)

    def run(sync):
        outs = []
        for i in range(12):
            x = sets[i % 3]
            outs.append([torch.full_like(x[0], float("nan")) for _ in range(3)])
            torch.cuda.synchronize()
        for i, out in enumerate(outs):
            fa.backward(*sets[i % 3], *out, b, h, s, d, scale, causal, dtype=dtype, workspace=ws, workspace_bytes=ws.numel(),
                        stream=torch.cuda.current_stream(dev))
            if sync:
                torch.cuda.synchronize()
                ws.fill_(255)                              # a delta read too early would be a NaN
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return outs

    ref = run(True)
    assert all(torch.isfinite(x.float()).all() for out in ref for x in out)
    for _ in range(3):
        for x, y in zip(run(False), ref):
            assert all(torch.equal(a, c) for a, c in zip(x, y))
    assert fa.device_status() == 0
