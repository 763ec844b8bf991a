"""Device KV cache objects (IKVCache surface) against the oracle: Update / Truncate / TrimToLast / Snapshot / Restore and
attention over an fp32 cache (KVCache + ScaledDotProductFlash*) and a Q8_0 cache (QuantizedKVCache +
ScaledDotProductFlashQ8_0*).

Q8_0 rows must be bit-exact with QuantizedKVCache.QuantizeRowQ8_0 (the snapshot speaks the reference's 34-byte block
layout, so it is compared byte for byte with the oracle's row quantiser); attention outputs within 1e-5 relative of the
oracle's restatement of the scalar flash kernels on the same (quantised) rows.
"""
import numpy as np
import pytest

from sharpmind_b200 import ops, synth
from tests.gpu_util import to_dev

pytestmark = pytest.mark.gpu


def _rows_q8(oracle, x):
    """x [..., headDim] fp32 -> [..., headDim/32*34] uint8, QuantizeRowQ8_0 per row."""
    hd = x.shape[-1]
    flat = x.reshape(-1, hd)
    q = oracle.quantize_rows_q8_0(flat, flat.shape[0], hd)
    return np.asarray(q, np.uint8).reshape(*x.shape[:-1], hd // 32 * 34)


def _oracle_attention(oracle, kind, q, kc, vc, length, scale):
    """q [B, S, H, D]; kc / vc [B, KVH, length, row] (fp32 rows or Q8_0 byte rows); returns [B, S, H, D]."""
    B, S, H, D = q.shape
    KVH = kc.shape[1]
    out = np.zeros_like(q)
    for b in range(B):
        for h in range(H):
            kh = h // (H // KVH)
            qq = np.ascontiguousarray(q[b, :, h, :])
            if kind == ops.KVCache.Q8_0:
                out[b, :, h, :] = oracle.sdpa_flash_q8(qq, kc[b, kh, :length], vc[b, kh, :length], scale)
            else:
                out[b, :, h, :] = oracle.sdpa_flash(qq, kc[b, kh, :length], vc[b, kh, :length], scale)
    return out


@pytest.mark.parametrize("kind", [ops.KVCache.F32, ops.KVCache.Q8_0])
@pytest.mark.parametrize("hd,heads,kvh", [(128, 8, 2), (64, 4, 4)])
def test_kv_cache_update_attention_truncate_snapshot(oracle, cuda, kind, hd, heads, kvh):
    B, max_seq = 2, 96
    kv = ops.KVCache(cuda, B, kvh, max_seq, hd, kind)
    assert kv.Length == 0 and kv.MaxSeqLen == max_seq and not kv.IsFull and kv.Snapshot() is None
    scale = 1.0 / np.sqrt(hd)
    # the oracle's cache: rows as the reference stores them
    row = hd // 32 * 34 if kind == ops.KVCache.Q8_0 else hd
    kc = np.zeros((B, kvh, max_seq, row), np.uint8 if kind == ops.KVCache.Q8_0 else np.float32)
    vc = np.zeros_like(kc)
    length = 0

    def append(tag, s):
        nonlocal length
        k = synth.normal("kv", f"k{tag}{hd}", (B, s, kvh, hd))
        v = synth.normal("kv", f"v{tag}{hd}", (B, s, kvh, hd))
        if tag == "z":
            k[:, 0, 0, :32] = 0.0  # an all-zero block takes d = 1
        kv.Update(to_dev(k), to_dev(v))
        kr, vr = (_rows_q8(oracle, k), _rows_q8(oracle, v)) if kind == ops.KVCache.Q8_0 else (k, v)
        kc[:, :, length:length + s] = kr.transpose(0, 2, 1, 3)
        vc[:, :, length:length + s] = vr.transpose(0, 2, 1, 3)
        length += s

    def check_attention(tag, s):
        q = synth.normal("kv", f"q{tag}{hd}", (B, s, heads, hd))
        got = kv.attention(to_dev(q), scale).cpu().numpy()
        want = _oracle_attention(oracle, kind, q, kc, vc, length, scale)
        assert np.max(np.abs(got - want)) <= 1e-5 * np.max(np.abs(want)), (tag, float(np.max(np.abs(got - want)) / np.max(np.abs(want))))

    append("a", 37)                 # a prompt chunk
    assert kv.Length == 37
    check_attention("a", 5)         # the last five positions as queries (several rows: prompt / verification shape)
    append("z", 1)
    check_attention("b", 1)         # one decode step
    # the stored rows are the reference's rows, byte for byte
    pos, sk, sv = kv.Snapshot()
    assert pos == length
    assert np.array_equal(sk.view(kc.dtype).reshape(B, kvh, length, row), kc[:, :, :length])
    assert np.array_equal(sv.view(vc.dtype).reshape(B, kvh, length, row), vc[:, :, :length])
    # speculative rollback: append draft positions, truncate them away, carry on
    snap = (pos, sk.copy(), sv.copy())
    saved_k, saved_v, saved_len = kc.copy(), vc.copy(), length
    append("d", 4)
    check_attention("d", 4)
    kv.Truncate(saved_len)
    kv.Truncate(saved_len + 100)    # never grows (Math.Min)
    assert kv.Length == saved_len
    kc, vc, length = saved_k, saved_v, saved_len
    append("e", 1)
    check_attention("e", 1)
    # Restore brings the snapshot back, on this object or a fresh one
    other = ops.KVCache(cuda, B, kvh, max_seq, hd, kind)
    other.Restore(snap)
    assert other.Length == saved_len
    kc2, vc2 = saved_k.copy(), saved_v.copy()
    q = synth.normal("kv", f"qr{hd}", (B, 1, heads, hd))
    got = other.attention(to_dev(q), scale).cpu().numpy()
    want = _oracle_attention(oracle, kind, q, kc2, vc2, saved_len, scale)
    assert np.max(np.abs(got - want)) <= 1e-5 * np.max(np.abs(want))
    other.Dispose()
    # sliding window: the last 20 positions move to the front
    kv.TrimToLast(20)
    assert kv.Length == 20
    kc[:, :, :20] = kc[:, :, length - 20:length].copy()
    vc[:, :, :20] = vc[:, :, length - 20:length].copy()
    length = 20
    check_attention("t", 1)
    kv.TrimToLast(50)               # keep >= length: nothing happens
    assert kv.Length == 20
    kv.Reset()
    assert kv.Length == 0
    # overflow is refused (KVCache.Update throws)
    with pytest.raises(ops.ArgumentOutOfRangeException):
        kv.Update(to_dev(np.zeros((B, max_seq + 1, kvh, hd), np.float32)), to_dev(np.zeros((B, max_seq + 1, kvh, hd), np.float32)))
    kv.Dispose()
    assert cuda.device_status() == 0


def test_q8_cache_long_context_decode(oracle, cuda):
    """The benchmark's context length: 2049 positions of a Q8_0 cache, 16 query heads over 8 cached heads."""
    B, kvh, heads, hd, n = 1, 8, 16, 128, 2049
    kv = ops.KVCache(cuda, B, kvh, n + 7, hd, ops.KVCache.Q8_0)
    k = synth.normal("kv", "klong", (B, n, kvh, hd))
    v = synth.normal("kv", "vlong", (B, n, kvh, hd))
    kv.Update(to_dev(k), to_dev(v))
    q = synth.normal("kv", "qlong", (B, 1, heads, hd))
    scale = 1.0 / np.sqrt(hd)
    got = kv.attention(to_dev(q), scale).cpu().numpy()
    kc, vc = _rows_q8(oracle, k).transpose(0, 2, 1, 3), _rows_q8(oracle, v).transpose(0, 2, 1, 3)
    want = _oracle_attention(oracle, ops.KVCache.Q8_0, q, np.ascontiguousarray(kc), np.ascontiguousarray(vc), n, scale)
    assert np.max(np.abs(got - want)) <= 1e-5 * np.max(np.abs(want))
    kv.Dispose()


@pytest.mark.parametrize("hd,heads,kvh", [(128, 8, 4), (128, 6, 2), (64, 4, 4), (64, 8, 1)])
def test_prompt_attention_on_tensor_cores(oracle, cuda, hd, heads, kvh):
    """Causal attention of a chunk of query rows over an fp32 cache with both contractions as bf16 MMAs on operands split
    three ways: within 1e-5 of the oracle's scalar flash attention (the bound of the fp32 kernel), for chunks that end
    inside a 64-row tile, start after an earlier chunk, and for query-head groups of 1, 2, 3 and 8; and the fp32
    CUDA-core kernel it replaces gives the same result to that bound."""
    B, max_seq = 2, 320
    kv = ops.KVCache(cuda, B, kvh, max_seq, hd, ops.KVCache.F32)
    scale = 1.0 / np.sqrt(hd)
    kc = np.zeros((B, kvh, max_seq, hd), np.float32)
    vc = np.zeros_like(kc)
    length = 0
    for tag, s in (("p", 150), ("q", 77), ("r", 1), ("s", 64)):
        k = synth.normal("kvmma", f"k{tag}{hd}", (B, s, kvh, hd))
        v = synth.normal("kvmma", f"v{tag}{hd}", (B, s, kvh, hd))
        if tag == "p":
            k *= 4.0  # sharper softmax: scores of a few units
        kv.Update(to_dev(k), to_dev(v))
        kc[:, :, length:length + s] = k.transpose(0, 2, 1, 3)
        vc[:, :, length:length + s] = v.transpose(0, 2, 1, 3)
        length += s
        q = synth.normal("kvmma", f"q{tag}{hd}", (B, s, heads, hd))
        got = kv.attention(to_dev(q), scale).cpu().numpy()
        want = _oracle_attention(oracle, ops.KVCache.F32, q, kc, vc, length, scale)
        err = float(np.max(np.abs(got - want)) / np.max(np.abs(want)))
        assert err <= 1e-5, (tag, err)
        if s > 1:
            cuda.set_option("prompt_attention_mma", 0)
            try:
                old = kv.attention(to_dev(q), scale).cpu().numpy()
            finally:
                cuda.set_option("prompt_attention_mma", 1)
            assert np.max(np.abs(old - got)) <= 2e-5 * np.max(np.abs(want))
            # one query head per CTA instead of two that share a KV head: every head's arithmetic is the same
            cuda.set_option("prompt_attention_heads_per_cta", 1)
            try:
                single = kv.attention(to_dev(q), scale).cpu().numpy()
            finally:
                cuda.set_option("prompt_attention_heads_per_cta", 0)
            assert np.array_equal(single.view(np.uint32), got.view(np.uint32))
    kv.Dispose()
    assert cuda.device_status() == 0


@pytest.mark.parametrize("hd,heads,kvh", [(128, 8, 4), (64, 6, 2)])
def test_prompt_attention_on_tensor_cores_over_a_q8_0_cache(oracle, cuda, hd, heads, kvh):
    """Chunks of 16 query rows and more over a Q8_0 cache take the tensor-core kernel with its K / V tiles staged as d * q
    (exact in the three bf16 parts): within 1e-5 of the oracle's ScaledDotProductFlashQ8_0 on the same quantised rows,
    and of the CUDA-core kernel it replaces; shorter chunks keep that kernel."""
    B, max_seq = 2, 320
    kv = ops.KVCache(cuda, B, kvh, max_seq, hd, ops.KVCache.Q8_0)
    scale = 1.0 / np.sqrt(hd)
    row = hd // 32 * 34
    kc = np.zeros((B, kvh, max_seq, row), np.uint8)
    vc = np.zeros_like(kc)
    length = 0
    for tag, s in (("p", 150), ("q", 77), ("r", 5), ("s", 64)):
        k = synth.normal("kvmmaq8", f"k{tag}{hd}", (B, s, kvh, hd))
        v = synth.normal("kvmmaq8", f"v{tag}{hd}", (B, s, kvh, hd))
        if tag == "p":
            k *= 4.0
        kv.Update(to_dev(k), to_dev(v))
        kc[:, :, length:length + s] = _rows_q8(oracle, k).transpose(0, 2, 1, 3)
        vc[:, :, length:length + s] = _rows_q8(oracle, v).transpose(0, 2, 1, 3)
        length += s
        q = synth.normal("kvmmaq8", f"q{tag}{hd}", (B, s, heads, hd))
        got = kv.attention(to_dev(q), scale).cpu().numpy()
        want = _oracle_attention(oracle, ops.KVCache.Q8_0, q, kc, vc, length, scale)
        err = float(np.max(np.abs(got - want)) / np.max(np.abs(want)))
        assert err <= 1e-5, (tag, err)
        cuda.set_option("prompt_attention_mma", 0)
        try:
            old = kv.attention(to_dev(q), scale).cpu().numpy()
        finally:
            cuda.set_option("prompt_attention_mma", 1)
        assert np.max(np.abs(old - got)) <= 2e-5 * np.max(np.abs(want))
        assert np.array_equal(old.view(np.uint32), got.view(np.uint32)) == (s < 16)  # which kernel ran
    kv.Dispose()
    assert cuda.device_status() == 0


@pytest.mark.parametrize("hd,heads,kvh,most", [(128, 32, 8, 3584), (128, 4, 2, 3584), (64, 8, 4, 1792)])
@pytest.mark.parametrize("rows,length", [(2, 97), (2, 98), (6, 128), (8, 129), (9, 257), (16, 1027), (5, 1700), (3, -1), (3, 0), (3, 1)])
def test_few_rows_over_a_long_cache(cuda, hd, heads, kvh, most, rows, length):
    """A draft's rows over an fp32 cache run on a cluster of CTAs per head pair: the same bits as the one-CTA walk (here reached
    by padding the same queries to 17 rows: a row's sums do not depend on the rows behind it), around the key tiles, with CTAs
    that get no tile, at the largest cache the cluster holds and past it (length counted from there when below 2).  Also against
    float64: an output is a convex combination of value rows whose weights are off by the scores' absolute error, a few
    roundings (2^-24) of the largest |q| |k| scale."""
    import torch

    length = length if length > 1 else most + length
    g = torch.Generator(device="cuda").manual_seed(rows * 7919 + length)
    pad = 17 - rows  # later positions, seen by the padding rows alone
    k, v = (torch.randn((1, length + pad, kvh, hd), generator=g, device="cuda") for _ in range(2))
    q = torch.randn((1, 17, heads, hd), generator=g, device="cuda")
    scale = hd ** -0.5
    kv = ops.KVCache(cuda, 1, kvh, length + pad, hd, ops.KVCache.F32)
    kv.Update(k, v)
    want = kv.attention(q, scale)[0, :rows]
    kv.Truncate(length)
    got = kv.attention(q[:, :rows].contiguous(), scale)[0]
    assert torch.equal(got.view(torch.int32), want.view(torch.int32)), int((got != want).sum())
    kd, vd = (t[0, :length].double().repeat_interleave(heads // kvh, 1).permute(1, 0, 2) for t in (k, v))
    s = q[0, :rows].double().permute(1, 0, 2) @ kd.transpose(1, 2) * scale
    pos = length - rows + torch.arange(rows, device="cuda")
    s = s.masked_fill(torch.arange(length, device="cuda")[None] > pos[:, None], -torch.inf)
    exact = (torch.softmax(s, -1) @ vd).permute(1, 0, 2)
    reach = float(q.norm(dim=-1).max() * k.norm(dim=-1).max()) * scale
    assert (got.double() - exact).abs().max() <= 4 * 2.0 ** -24 * reach * v.abs().max()
    kv.Dispose()


@pytest.mark.parametrize("hd,group,resident", [(128, 2, 3), (128, 1, 4), (64, 2, 5), (64, 1, 7)])
@pytest.mark.parametrize("kind", [ops.KVCache.F32, ops.KVCache.Q8_0])
@pytest.mark.parametrize("length", [1, 17, 40, 64])
def test_decode_attention_forms_keep_the_bits(cuda, hd, group, resident, kind, length):
    """One sequence's decode attention by the number of CTAs that the grid has: with and without keys requested ahead, on both sides of
    the lines between the forms (`resident` CTAs per SM with look-ahead).  Up to 64 positions a CTA takes a whole cached head whatever
    the batch, so every batch gives a sequence the same bits, and the ones of small batches are right (float64, a few roundings
    of weights and sums)."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = 7 * sms + 1
    g = torch.Generator(device="cuda").manual_seed(hd + group + length)
    k, v = (torch.randn((most, length, 1, hd), generator=g, device="cuda") for _ in range(2))
    q = torch.randn((most, 1, group, hd), generator=g, device="cuda")

    def attend(lo, hi):
        kv = ops.KVCache(cuda, hi - lo, 1, length, hd, kind)
        kv.Update(k[lo:hi].contiguous(), v[lo:hi].contiguous())
        out = kv.attention(q[lo:hi].contiguous(), hd ** -0.5)
        torch.cuda.synchronize()
        kv.Dispose()
        return out

    want = torch.cat([attend(lo, min(lo + 64, most)) for lo in range(0, most, 64)])
    for n in sorted({resident * sms, resident * sms + 1, 4 * sms + 1, 6 * sms + 1, most}):
        got = attend(0, n)
        assert torch.equal(got.view(torch.int32), want[:n].view(torch.int32)), n
    if kind == ops.KVCache.F32:
        p = torch.softmax(torch.einsum("bgd,bld->bgl", q[:, 0].double(), k[:, :, 0].double()) * hd ** -0.5, -1)
        exact = torch.einsum("bgl,bld->bgd", p, v[:, :, 0].double())
        reach = float(q.norm(dim=-1).max() * k.norm(dim=-1).max()) * hd ** -0.5
        assert (want[:, 0].double() - exact).abs().max() <= 4 * 2.0 ** -24 * max(reach, 8.0) * v.abs().max()


@pytest.mark.parametrize("kind", ["f32", "q8_0"])
@pytest.mark.parametrize("hd,heads,kvh", [(128, 4, 2), (64, 3, 1)])
def test_prompt_attention_on_tcgen05_gives_the_bits_of_mma_sync(cuda, kind, hd, heads, kvh):
    """The tcgen05 kernel against the mma.sync kernel (one head per CTA selects it), bit for bit: lengths at the borders of its key tiles
    (32), chunks (64) and row tiles (128), starts that are no multiple of any, enough chunks for every barrier to go round, and scores that
    keep raising the running maximum."""
    import torch

    scale = 1.0 / np.sqrt(hd)
    for n0, s in ((0, 33), (0, 64), (31, 34), (0, 127), (0, 128), (0, 129), (17, 175), (70, 58), (500, 260), (1003, 18)):
        kv = ops.KVCache(cuda, 1, kvh, n0 + s, hd, ops.KVCache.Q8_0 if kind == "q8_0" else ops.KVCache.F32)
        ramp = np.linspace(0.2, 4.0, n0 + s, dtype=np.float32)[None, :, None, None]
        k = to_dev(synth.normal("kvtc", f"k{hd}{n0}{s}", (1, n0 + s, kvh, hd)) * ramp)
        v = to_dev(synth.normal("kvtc", f"v{hd}{n0}{s}", (1, n0 + s, kvh, hd)))
        if n0:
            kv.Update(k[:, :n0].contiguous(), v[:, :n0].contiguous())
        kv.Update(k[:, n0:].contiguous(), v[:, n0:].contiguous())
        q = to_dev(synth.normal("kvtc", f"q{hd}{n0}{s}", (1, s, heads, hd)) * 2.0)
        got = kv.attention(q, scale)
        cuda.set_option("prompt_attention_heads_per_cta", 1)
        try:
            want = kv.attention(q, scale)
        finally:
            cuda.set_option("prompt_attention_heads_per_cta", 0)
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (n0, s)
        kv.Dispose()
    assert cuda.device_status() == 0


def test_prompt_attention_first_called_under_capture():
    """The object's planes are allocated by its first call, a captured one too: the bits of an eager call, here and replayed after longer ones."""
    import torch

    ctx = ops.CudaContext(0)
    kv = ops.KVCache(ctx, 1, 2, 200, 128, ops.KVCache.F32)
    kv.Update(*(to_dev(synth.normal("kvcap", n, (1, 200, 2, 128))) for n in "kv"))
    q = to_dev(synth.normal("kvcap", "q", (1, 150, 4, 128)))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = kv.attention(q, 128 ** -0.5)
    graph.replay()
    torch.cuda.synchronize()
    want = kv.attention(q, 128 ** -0.5)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    other = ops.KVCache(ctx, 1, 2, 2000, 128, ops.KVCache.F32)
    other.Update(*(to_dev(synth.normal("kvcap", "o" + n, (1, 2000, 2, 128))) for n in "kv"))
    other.attention(to_dev(synth.normal("kvcap", "oq", (1, 300, 4, 128))), 128 ** -0.5)
    got.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert ctx.device_status() == 0
    graph.reset()
    kv.Dispose(), other.Dispose()
    ctx.close()


@pytest.mark.parametrize("kind", ["f32", "q8_0"])
def test_prompt_attention_of_two_caches_on_two_streams(cuda, kind):
    """Two cache objects of one context, each on a stream of its own, their calls interleaved without a wait: the bits that each gives alone."""
    import torch

    shapes = [(700, 190), (650, 150)]  # positions, query rows
    caches, queries, want = [], [], []
    for i, (n, s) in enumerate(shapes):
        kv = ops.KVCache(cuda, 2, 2, n, 128, ops.KVCache.Q8_0 if kind == "q8_0" else ops.KVCache.F32)
        kv.Update(*(to_dev(synth.normal("kv2s", f"{x}{i}", (2, n, 2, 128))) for x in "kv"))
        caches.append(kv), queries.append(to_dev(synth.normal("kv2s", f"q{i}", (2, s, 4, 128))))
        want.append(kv.attention(queries[i], 128 ** -0.5))
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], [[], []]
    for _ in range(30):
        for i in (0, 1):
            with torch.cuda.stream(streams[i]):
                got[i].append(caches[i].attention(queries[i], 128 ** -0.5))
    torch.cuda.synchronize()
    for i in (0, 1):
        assert all(torch.equal(g.view(torch.int32), want[i].view(torch.int32)) for g in got[i]), i
        caches[i].Dispose()
    assert cuda.device_status() == 0


def test_prompt_attention_allocates_once_per_cache():
    """The first call over several rows takes room for all positions; the device's free memory stays what it is over the rest of the prompt."""
    import torch

    n, s, ctx = 4096, 512, ops.CudaContext(0)
    kv = ops.KVCache(ctx, 1, 8, n, 128, ops.KVCache.F32)
    k, v = (to_dev(synth.normal("kvone", x, (1, n, 8, 128))) for x in "kv")
    q = to_dev(synth.normal("kvone", "q", (1, s, 16, 128)))
    free = []
    for start in range(0, n, s):
        kv.Update(k[:, start:start + s].contiguous(), v[:, start:start + s].contiguous())
        kv.attention(q, 128 ** -0.5)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert len(set(free)) == 1, free
    kv.Dispose()
    ctx.close()


def _prompt_model(oracle, ctx, kv_dtype, max_seq, kv_heads=2):
    from sharpmind_b200.decoder import Decoder

    cfg = dict(n_layers=2, hidden=256, n_heads=kv_heads * 2, n_kv_heads=kv_heads, head_dim=128, ffn=512, vocab=1024, max_seq=max_seq, dtype=8, eps=1e-6,
               rope_theta=1.0e6, neox=True, qk_norm=True, kv_dtype=kv_dtype)
    return Decoder(ctx, cfg, synth.make_decoder_weights(cfg, "kvprompt", oracle.quantize), max_batch=1)


@pytest.mark.parametrize("kv_dtype", [0, 8])
def test_prompt_in_chunks_allocates_nothing(oracle, kv_dtype):
    """After the first chunk (activation rows) no chunk of a prompt allocates: the attention's planes are there from the model's creation."""
    import torch

    n, chunk, ctx = 4096, 256, ops.CudaContext(0)
    dec = _prompt_model(oracle, ctx, kv_dtype, n, kv_heads=16)
    tokens = torch.from_numpy(synth.token_ids("kvprompt", "chunks", (n,), 1024)).cuda()
    free = []
    for start in range(0, n, chunk):
        dec.forward_last_logits(tokens[start:start + chunk], pos=start)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert len(set(free)) == 1, free
    dec.close()
    ctx.close()


@pytest.mark.parametrize("kv_dtype", [0, 8])
def test_captured_prompt_pass_outlives_longer_contexts(oracle, cuda, kv_dtype):
    """A captured prompt pass replayed after eager passes further into the cache, of this model and of a larger one: the same logits."""
    import torch

    n = 256
    dec, big = _prompt_model(oracle, cuda, kv_dtype, 1024), _prompt_model(oracle, cuda, kv_dtype, 4096)
    tokens = torch.from_numpy(synth.token_ids("kvprompt", "cap", (1024,), 1024)).cuda()
    first = tokens[:n].contiguous()
    want = dec.forward_last_logits(first)[0].clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got, _ = dec.forward_last_logits(first)
    for pos in (n, 2 * n, 3 * n):
        dec.forward_last_logits(tokens[pos:pos + n], pos=pos)
    big.forward_last_logits(tokens[:n], pos=3000)
    torch.cuda.synchronize()
    got.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert cuda.device_status() == 0
    graph.reset()
    dec.close(), big.close()


@pytest.mark.parametrize("kind", ["f32", "q8_0"])
@pytest.mark.parametrize("hd,heads,kvh", [(128, 4, 2), (64, 4, 1), (64, 3, 1)])
def test_prompt_attention_off_16_byte_outputs(cuda, kind, hd, heads, kvh):
    """Outputs that the tcgen05 kernel does not take (8 bytes off a multiple of 16) go to the mma.sync kernel, two heads per CTA where they share a
    KV head: the same bits, over several key tiles and row tiles."""
    import torch

    for n0, s in ((0, 130), (77, 100)):
        kv = ops.KVCache(cuda, 1, kvh, n0 + s, hd, ops.KVCache.Q8_0 if kind == "q8_0" else ops.KVCache.F32)
        kv.Update(*(to_dev(synth.normal("kvoff", f"{x}{hd}{s}", (1, n0 + s, kvh, hd))) for x in "kv"))
        q = to_dev(synth.normal("kvoff", f"q{hd}{s}", (1, s, heads, hd)))
        want = kv.attention(q, hd ** -0.5)
        room = torch.empty(q.numel() + 4, dtype=torch.float32, device="cuda")
        got = room[2:2 + q.numel()]
        cuda.check(cuda.lib.smc_sdpa_kv_dev(cuda.h, kv.h, q.data_ptr(), got.data_ptr(), 1, heads, s, hd ** -0.5, kv._stream()))
        assert torch.equal(got.view(torch.int32), want.flatten().view(torch.int32)), (n0, s)
        kv.Dispose()


def test_decode_attention_keeps_its_speed_behind_a_staged_matmul(cuda):
    """A matmul whose operands fill shared memory leaves the SMs little L1; the fp32 decode attention behind it lives on L1.  32 sequences: behind the
    matmul it takes at most 1.5 times what it takes alone (2.4 times where it does not ask for its L1)."""
    import torch

    from sharpmind_b200.ops import Mode

    n, dev = 2048, ops.DeviceOps(cuda)
    g = torch.Generator(device="cuda").manual_seed(3)
    kv = ops.KVCache(cuda, 32, 8, n, 128, ops.KVCache.F32)
    kv.Update(*(torch.randn((32, n, 8, 128), generator=g, device="cuda") for _ in "kv"))
    q = torch.randn((32, 1, 16, 128), generator=g, device="cuda")
    w = cuda.register_dev(dev.quantize_weights(8, torch.randn((6144, 1024), generator=g, device="cuda") * 0.02), 8, 6144, 1024)
    x = torch.randn((32, 1024), generator=g, device="cuda")

    def both():
        dev.qmatmul(x, w, Mode.ACT_Q8)
        kv.attention(q, 128 ** -0.5)

    def us(f):
        times = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                f()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 50.0)
        return min(times[1:])

    alone, behind, matmul = us(lambda: kv.attention(q, 128 ** -0.5)), us(both), us(lambda: dev.qmatmul(x, w, Mode.ACT_Q8))
    assert behind - matmul <= 1.5 * alone, (alone, behind, matmul)
    cuda.release(w)
    kv.Dispose()
