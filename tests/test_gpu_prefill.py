"""Prefill-sized Q4_K matmul on the tensor cores against the oracle's scalar vec-dot (fp32 activations).

Bound: 1e-5 * ||w_row|| * ||x_row|| per output, the same as the fp32-activation GEMV: the tensor-core path
multiplies exact integer weight parts with an fp16 (hi, lo) split of the activations.
"""
import numpy as np
import pytest

from sharpmind_b200 import ops, synth
from tests.gpu_util import Q4_K, Q6_K, row_norm_bound, to_dev

pytestmark = pytest.mark.gpu


def _case(oracle, cuda, dev, n, k, m, sigma_x=1.0, tag=""):
    wf = synth.normal("prefill", f"w{n}x{k}{tag}", (n, k), 0.02)
    raw = oracle.quantize(Q4_K, wf)
    x = synth.normal("prefill", f"x{m}x{k}{tag}", (m, k), sigma_x)
    w = cuda.register(raw, Q4_K, n, k)
    got = dev.qmatmul_tc(to_dev(x), w).cpu().numpy()
    assert cuda.device_status() == 0
    return raw, x, got, w


@pytest.mark.parametrize("n,k,m", [
    (128, 256, 128),     # one tile, one block
    (128, 1024, 128),    # several blocks: both accumulator buffers, stage reuse
    (256, 2048, 200),    # two row tiles, ragged token tile
    (384, 512, 1),       # a single token
    (128, 4096, 300),    # three token tiles
])
def test_tc_matmul_matches_oracle(oracle, cuda, dev, n, k, m):
    raw, x, got, w = _case(oracle, cuda, dev, n, k, m)
    want = oracle.qmatmul(Q4_K, x, raw, m, k, n)
    bound = row_norm_bound(oracle, Q4_K, raw, n, k, x)
    err = np.abs(got - want)
    assert np.all(err <= bound), float(np.max(err / bound))
    cuda.release(w)


@pytest.mark.parametrize("size", [1e-37, 1e-40, 3e37])
def test_tc_matmul_rows_at_the_ends_of_the_range(oracle, cuda, dev, size):
    """Rows whose scale would have no finite inverse, and very large ones: the bound of the mode at the row's own size, and a few
    of fp32's smallest numbers where the sums fall below its normal range."""
    n, k, m = 128, 512, 130
    raw = oracle.quantize(Q4_K, synth.normal("prefill", "wends", (n, k), 0.02))
    x = synth.normal("prefill", "xends", (m, k))
    x[::3] = (x[::3].astype(np.float64) * size).astype(np.float32)
    w = cuda.register(raw, Q4_K, n, k)
    got = dev.qmatmul_tc(to_dev(x), w).cpu().numpy()
    want = x.astype(np.float64) @ oracle.dequantize(Q4_K, raw, n * k).reshape(n, k).astype(np.float64).T
    bound = row_norm_bound(oracle, Q4_K, raw, n, k, x) + k * 2.0 ** -149
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))
    cuda.release(w)


@pytest.mark.parametrize("n,k", [(28672, 8192), (8192, 28672)])
def test_tc_matmul_llama70b_shapes_sampled_rows(oracle, cuda, dev, n, k):
    """The benchmarked prefill shapes (Llama-3-70B FFN, 512 tokens): weights drawn and quantised on the device, sampled
    weight rows (first, last, both sides of a 128-row tile edge, 16 random ones) against the oracle's scalar vec-dot
    on every token, at the same per-output bound as the small shapes (the bound scales with ||w|| ||x||, hence with K)."""
    import torch

    m = 512
    g = torch.Generator(device="cuda").manual_seed(n + 7 * k)
    raw_d = dev.quantize_weights(Q4_K, torch.randn((n, k), generator=g, device="cuda") * 0.02)
    w = cuda.register_dev(raw_d, Q4_K, n, k)
    x = synth.normal("prefill", f"x70b_{k}", (m, k))
    got = dev.qmatmul_tc(to_dev(x), w).cpu().numpy()
    assert cuda.device_status() == 0
    rs = np.random.default_rng(n)
    rows = sorted({0, n - 1, 127, 128, n // 2 - 1, n // 2} | set(int(r) for r in rs.integers(0, n, 16)))
    per_row = k // 256 * 144
    xn = np.linalg.norm(x.astype(np.float64), axis=1)
    worst = 0.0
    for r in rows:
        raw_row = raw_d[r * per_row:(r + 1) * per_row].cpu().numpy()
        want = oracle.qmatmul(Q4_K, x, raw_row, m, k, 1)[:, 0]
        wn = np.linalg.norm(oracle.dequantize(Q4_K, raw_row, k).astype(np.float64))
        bound = 1e-5 * wn * xn
        err = np.abs(got[:, r].astype(np.float64) - want)
        worst = max(worst, float(np.max(err / bound)))
        assert np.all(err <= bound), (r, worst)
    print(f"tcgen05 matmul {n}x{k}, 512 tokens: worst error {worst:.3f} of the bound over {len(rows)} sampled rows")
    cuda.release(w)


def test_tc_matmul_scaling_and_zero_rows(oracle, cuda, dev):
    """Rows of very different magnitude (per-token power-of-two scale) and an all-zero row."""
    n, k, m = 128, 512, 16
    wf = synth.normal("prefill", "wz", (n, k), 0.02)
    raw = oracle.quantize(Q4_K, wf)
    x = synth.normal("prefill", "xz", (m, k))
    x[1] *= 1e-6
    x[2] *= 3e5
    x[3] = 0.0
    w = cuda.register(raw, Q4_K, n, k)
    got = dev.qmatmul_tc(to_dev(x), w).cpu().numpy()
    want = oracle.qmatmul(Q4_K, x, raw, m, k, n)
    bound = row_norm_bound(oracle, Q4_K, raw, n, k, x)
    assert np.all(np.abs(got - want) <= bound + 1e-30)
    assert np.all(got[3] == 0.0)
    cuda.release(w)


def test_tc_matmul_agrees_with_gemv_path(oracle, cuda, dev):
    n, k, m = 256, 1024, 64
    raw, x, got, w = _case(oracle, cuda, dev, n, k, m, tag="g")
    ref = dev.qmatmul(to_dev(x), w, ops.Mode.ACT_F32).cpu().numpy()
    bound = 2 * row_norm_bound(oracle, Q4_K, raw, n, k, x)
    assert np.all(np.abs(got - ref) <= bound)
    cuda.release(w)


def test_tc_matmul_rejects_other_shapes(oracle, cuda, dev):
    raw = oracle.quantize(Q4_K, synth.normal("prefill", "wr", (64, 256), 0.02))
    w = cuda.register(raw, Q4_K, 64, 256)
    with pytest.raises(ops.NotSupportedException):
        dev.qmatmul_tc(to_dev(synth.normal("prefill", "xr", (4, 256))), w)
    cuda.release(w)


@pytest.mark.parametrize("n,k,m", [(256, 2048, 64), (128, 4096, 300), (384, 1024, 129)])
def test_quantised_activations_at_prefill_sizes_run_on_the_tensor_cores(oracle, cuda, dev, n, k, m):
    """SMC_ACT_Q8 over Q4_K at 64 rows and more: the Q8_0 activation rows go through the tcgen05 kernel (d * q is exact in
    its fp16 pairs).  Against the oracle on the dequantised rows at the mode's bound; against the int8 kernels of the same
    library (option off) to a few ulps of the row scale; and the two entry points (fp32 rows in, Q8 rows in) bit for bit."""
    raw = oracle.quantize(Q4_K, synth.normal("prefill", f"wq{n}x{k}", (n, k), 0.02))
    x = synth.normal("prefill", f"xq{m}x{k}", (m, k))
    w = cuda.register(raw, Q4_K, n, k)
    xd = to_dev(x)
    got = dev.qmatmul(xd, w, ops.Mode.ACT_Q8).cpu().numpy()
    xq = oracle.quantize_rows_q8_0(x, m, k)
    from tests.gpu_util import Q8_0
    xhat = np.stack([oracle.dequantize(Q8_0, xq[r], k) for r in range(m)])
    want = oracle.qmatmul(Q4_K, xhat, raw, m, k, n)
    bound = row_norm_bound(oracle, Q4_K, raw, n, k, xhat)
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))
    act = ops.Q8Act(cuda, m, k)
    dev.quantize_q8(xd, act, k)
    assert np.array_equal(dev.qmatmul_q8(act, w).cpu().numpy().view(np.uint32), got.view(np.uint32))
    cuda.set_option("q8_prefill_tensor_cores", 0)
    try:
        ints = dev.qmatmul_q8(act, w).cpu().numpy()
    finally:
        cuda.set_option("q8_prefill_tensor_cores", 1)
    assert np.all(np.abs(ints - got) <= bound)
    act.close()
    cuda.release(w)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("n,k,m", [
    (7936, 256, 64),     # one block, half a token tile, the fewest outputs that come this way
    (3968, 768, 128),    # rows that start inside a unit of eight blocks, fewer blocks than are folded at once
    (3968, 2048, 129),   # a token tile of one
    (2560, 4352, 200),   # 17 blocks: a last chain of one block
    (8192, 1024, 300),   # two waves of tiles
])
def test_q6k_fp32_rows_on_the_tensor_cores(oracle, cuda, dev, n, k, m):
    """fp32 rows over Q6_K at 64 rows and more: the weights' integer parts reach 4096 and travel as exact bfloat16 pairs.  Scales of
    every size and sign (products above 256 need the second half of the pair), rows of very different magnitude (one whose
    scale has no finite inverse) and a zero row;
    against float64 over the dequantised weights at the bound of the mode, and no further off than the digit planes it replaces.
    A row has the same bits whatever the batch it travels in, as long as that batch comes this way too."""
    import torch

    rs = np.random.default_rng(n + k + m)
    raw = np.array(oracle.quantize(Q6_K, synth.normal("prefill", f"w6{n}x{k}", (n, k), 0.02)), np.uint8).reshape(-1, 210)
    raw[:, 192:208] = rs.integers(0, 256, (raw.shape[0], 16), dtype=np.uint8)
    raw = np.ascontiguousarray(raw.reshape(-1))
    x = synth.normal("prefill", f"x6{m}x{k}", (m, k))
    x[1] *= 1e-6
    x[2] *= 3e5
    x[3] = 0.0
    x[4] *= 1e-37
    w = cuda.register(raw, Q6_K, n, k)
    got = dev.qmatmul(to_dev(x), w, ops.Mode.ACT_F32).cpu().numpy()
    assert cuda.device_status() == 0
    want = x.astype(np.float64) @ oracle.dequantize(Q6_K, raw, n * k).reshape(n, k).astype(np.float64).T
    bound = row_norm_bound(oracle, Q6_K, raw, n, k, x)
    bound += k * 2.0 ** -149  # sums of the smallest row round at fp32's smallest number
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))
    assert np.all(got[3] == 0.0)
    more = np.concatenate([x[5:37], x])  # other neighbours, another place in the tile, more rows
    again = dev.qmatmul(to_dev(more), w, ops.Mode.ACT_F32).cpu().numpy()
    assert np.array_equal(again[32:].view(np.uint32), got.view(np.uint32)) and np.array_equal(again[:32].view(np.uint32), got[5:37].view(np.uint32))
    # the digit planes take batches below 64 rows
    planes = torch.cat([dev.qmatmul(to_dev(x[i:i + 32]), w, ops.Mode.ACT_F32) for i in range(0, m, 32)]).cpu().numpy()
    live = [i for i in range(m) if i not in (3, 4)]  # row 4: the planes' own scales fall below fp32's normal range
    err = [float(np.linalg.norm(((y - want) / np.linalg.norm(want, axis=1, keepdims=True).clip(1e-30))[live])) for y in (got, planes)]
    print(f"{n}x{k}, {m} rows: error {err[0]:.2e}, digit planes {err[1]:.2e}")
    assert err[0] <= err[1]
    cuda.release(w)


def test_host_threads_on_one_context_and_stream(oracle):
    """Matmuls that keep an image of their rows in the context, queued by several host threads on one stream: every result
    has the bits of the same call made alone (no thread's image is overwritten before its contraction is queued, and no
    buffer is freed under a call when another thread's larger one grows it; the sizes grow as the threads go on)."""
    import threading

    import torch

    cases = []
    raw4 = oracle.quantize(Q4_K, synth.normal("threads", "w4", (256, 512), 0.02))
    raw6 = oracle.quantize(Q6_K, synth.normal("threads", "w6", (7936, 256), 0.02))
    wb = synth.normal("threads", "wb", (256, 512), 0.02)

    def weights(ctx):
        b = torch.from_numpy(wb).cuda().to(torch.bfloat16).view(torch.uint8).reshape(-1)
        return {"q4": ctx.register(raw4, Q4_K, 256, 512), "q6": ctx.register(raw6, Q6_K, 7936, 256),
                "bf16": ctx.register_dev(b, ops.QuantDType.BF16, 256, 512, repack=False)}

    for name, k, mode in (("q4", 512, ops.Mode.ACT_F32), ("q6", 256, ops.Mode.ACT_F32), ("q4", 512, ops.Mode.ACT_Q8), ("bf16", 512, ops.Mode.ACT_BF16)):
        cases.append((name, mode, [to_dev(synth.normal("threads", f"x{name}{int(mode)}{m}", (m, k))) for m in (64, 70, 128, 190, 256, 391)]))

    def run_all(threads):
        ctx = ops.CudaContext(0)
        dev, w = ops.DeviceOps(ctx), weights(ctx)
        torch.cuda.synchronize()
        out, failed = [[] for _ in cases], []

        def body(i):
            name, mode, xs = cases[i]
            try:
                for x in xs:
                    y = [dev.qmatmul(x, w[name], mode) for _ in range(24)]
                    out[i] += y + [dev.argmax(t) for t in y[::8]]
            except Exception as e:  # reported below, by the test's own thread
                failed.append(e)

        if threads:
            ts = [threading.Thread(target=body, args=(i,)) for i in range(len(cases))]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
        else:
            for i in range(len(cases)):
                body(i)
        torch.cuda.synchronize()
        assert not failed, failed
        assert ctx.device_status() == 0
        for h in w.values():
            ctx.release(h)
        ctx.close()
        return out

    alone, together = run_all(False), run_all(True)
    for (name, mode, xs), a, b in zip(cases, alone, together):
        wrong = [i for i, (u, v) in enumerate(zip(a, b)) if not torch.equal(u.view(torch.int32), v.view(torch.int32))]
        assert not wrong, (name, mode, wrong)


def _capture(body):
    """Captures `body` and replays the graph."""
    import torch

    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        body()
    g.replay()
    torch.cuda.synchronize()
    return g


@pytest.mark.parametrize("warm,then", [
    ((200, 3584, 256), [(200, 3584, 256), (140, 3584, 256), (139, 3584, 256), (64, 3584, 256), (2, 3584, 256)]),  # both sides of the line between the forms
    ((63, 8192, 512), [(64, 7936, 256), (63, 8192, 512)]),   # first the digit planes
    ((201, 2560, 4352), [(129, 3968, 6656)]),                # fewer values, but as many tiles of rows of a longer K
])
def test_fp32_rows_over_q6k_reserve_for_both_forms(oracle, warm, then):
    """SMC_ACT_F32 over Q6_K takes one of two forms by M and N.  A call with no more values and no more outputs than an earlier
    one does not allocate, whichever forms the two take: it can be captured."""
    import torch

    ctx = ops.CudaContext(0)
    dev, ws = ops.DeviceOps(ctx), {}
    for m, n, k in [warm] + then:
        if (n, k) not in ws:
            ws[n, k] = ctx.register(oracle.quantize(Q6_K, synth.normal("both", f"w{n}x{k}", (n, k), 0.02)), Q6_K, n, k)

    def call(m, n, k):
        return dev.qmatmul(to_dev(synth.normal("both", f"x{m}x{k}", (m, k))), ws[n, k], ops.Mode.ACT_F32)

    call(*warm)
    xs = [to_dev(synth.normal("both", f"x{m}x{k}", (m, k))) for m, n, k in then]
    outs = [torch.empty((m, n), device="cuda") for m, n, k in then]
    g = _capture(lambda: [dev.qmatmul(x, ws[n, k], ops.Mode.ACT_F32, out=o) for x, o, (m, n, k) in zip(xs, outs, then)])
    for o, c in zip(outs, then):
        assert torch.equal(o, call(*c)), c
    del g
    for w in ws.values():
        ctx.release(w)
    assert ctx.device_status() == 0
    ctx.close()


@pytest.mark.parametrize("outlier", [1e4, 1e5, 1e12, 1e30])
def test_q6k_fp32_rows_with_an_element_far_above_the_others(oracle, cuda, dev, outlier):
    """A row's largest element lies where the weights are zero: the others keep the accuracy that they have in the digit planes,
    whose scales are per 32 elements.  Bounds as in test_q6k_fp32_rows_on_the_tensor_cores."""
    import torch

    n, k, m = 3968, 768, 129
    raw = np.array(oracle.quantize(Q6_K, synth.normal("prefill", f"w6o{n}x{k}", (n, k), 0.02)), np.uint8).reshape(n, k // 256, 210)
    raw[:, 1, 192 + 4:192 + 6] = 0  # scales of elements 64 .. 95 of the second block
    raw = np.ascontiguousarray(raw.reshape(-1))
    x = synth.normal("prefill", f"x6o{m}x{k}", (m, k))
    rest = x.copy()
    rest[:, 256 + 64:256 + 96] = 0.0
    x[::2, 256 + 70] = outlier
    w = cuda.register(raw, Q6_K, n, k)
    got = dev.qmatmul(to_dev(x), w, ops.Mode.ACT_F32).cpu().numpy()
    planes = torch.cat([dev.qmatmul(to_dev(x[i:i + 32]), w, ops.Mode.ACT_F32) for i in range(0, m - 1, 32)]).cpu().numpy()
    assert cuda.device_status() == 0
    want = x.astype(np.float64) @ oracle.dequantize(Q6_K, raw, n * k).reshape(n, k).astype(np.float64).T
    bound = row_norm_bound(oracle, Q6_K, raw, n, k, rest)  # the outlier does not widen it
    assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))
    err = [float(np.linalg.norm((y - want[:m - 1]) / np.linalg.norm(want[:m - 1], axis=1, keepdims=True))) for y in (got[:m - 1], planes)]
    print(f"outlier {outlier:.0e}: error {err[0]:.2e}, digit planes {err[1]:.2e}")
    assert err[0] <= err[1]
    cuda.release(w)
