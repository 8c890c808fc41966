"""GPU parity of the two multi-query attention kernels, each forced in turn: the tcgen05 kernel
(option attn_tc = 1) and the mma.sync kernel (attn_tc = 0), against the oracle's
multiMasklessSDPA / multiMaskedSDPA restatements (attention.zig:125-234, 416-541)."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_close_ref, f16_normal

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 0], ids=["tcgen05", "mma_sync"])
def forced(ctx, request):
    ctx.set_option("attn_tc", request.param)
    yield request.param
    ctx.set_option("attn_tc", -1)


@pytest.mark.parametrize("h,lq,lk,d", [(16, 729, 729, 72), (2, 5, 5, 72), (3, 37, 53, 72), (4, 170, 170, 64),
                                       (2, 128, 64, 64), (2, 129, 65, 64), (1, 1, 1, 64), (3, 257, 1000, 72),
                                       (1, 300, 2048, 64)])
def test_maskless(ctx, oracle, forced, h, lq, lk, d):
    rng = np.random.default_rng(lq * 7 + lk + d)
    q, k, v = f16_normal(rng, (h, lq, d)), f16_normal(rng, (h, lk, d)), f16_normal(rng, (h, lk, d))
    assert_close_ref(ctx.sdpa_maskless(q, k, v, h, lq, lk, d), oracle.sdpa_maskless(q, k, v), "maskless")


@pytest.mark.parametrize("pos,s", [(0, 1), (0, 7), (16, 37), (0, 761), (300, 70), (63, 130), (1000, 129)])
def test_causal_mask(ctx, oracle, forced, pos, s):
    m = ctx.create_attention_mask(pos, s)
    rng = np.random.default_rng(pos + s)
    h = 32 if s < 100 else 4
    q, k, v = f16_normal(rng, (h, s, 64)), f16_normal(rng, (h, pos + s, 64)), f16_normal(rng, (h, pos + s, 64))
    assert_close_ref(ctx.sdpa_masked(q, k, v, m, h, s, pos + s, 64), oracle.sdpa_masked(q, k, v, m), "masked")


def test_arbitrary_mask(ctx, oracle, forced):
    rng = np.random.default_rng(12)
    q, k, v = f16_normal(rng, (4, 150, 64)), f16_normal(rng, (4, 190, 64)), f16_normal(rng, (4, 190, 64))
    m = (rng.random((150, 190)) > 0.3).astype(np.uint8)
    m[:, 0] = 1  # every row keeps at least one key
    assert_close_ref(ctx.sdpa_masked(q, k, v, m, 4, 150, 190, 64), oracle.sdpa_masked(q, k, v, m), "random mask")


@pytest.mark.parametrize("h,lq,lk,lo,hi", [(2, 129, 65, 64, 65), (3, 65, 300, 70, 131), (2, 200, 640, 0, 64), (1, 256, 1000, 999, 1000),
                                           (2, 384, 257, 100, 257)])
def test_mask_whose_tiles_are_partly_unseen(ctx, oracle, forced, h, lq, lk, lo, hi):
    """Rows see some of the keys lo..hi, one row in every 128 nothing (zeros), the second query block (where there is one)
    a single key: tiles before, between and after are skipped by the tcgen05 kernel."""
    rng = np.random.default_rng(lq + lk)
    q, k, v = f16_normal(rng, (h, lq, 64)), f16_normal(rng, (h, lk, 64)), f16_normal(rng, (h, lk, 64))
    m = np.zeros((lq, lk), np.uint8)
    m[:, lo:hi] = rng.integers(0, 256, (lq, hi - lo)) * (rng.random((lq, hi - lo)) > 0.3)
    m[:, hi - 1] = 7        # any byte but 0 means visible
    m[128:256] = 0
    m[128:256, lo] = 1
    m[5::128] = 0
    got = ctx.sdpa_masked(q, k, v, m, h, lq, lk, 64)
    seen = m.any(1)
    assert (got[:, ~seen] == 0).all()
    ref = oracle.sdpa_masked(q, k, v, (m != 0).astype(np.uint8))
    assert_close_ref(got[:, seen], ref[:, seen], "partly unseen")


def test_large_scores_stay_finite(ctx, oracle, forced):
    """Scores far from zero: the running-max rescale must keep exp() in range in every tile."""
    rng = np.random.default_rng(5)
    q, k, v = f16_normal(rng, (2, 200, 64), 6.0), f16_normal(rng, (2, 300, 64), 6.0), f16_normal(rng, (2, 300, 64))
    got = ctx.sdpa_maskless(q, k, v, 2, 200, 300, 64)
    assert np.isfinite(got.astype(np.float32)).all()
    assert_close_ref(got, oracle.sdpa_maskless(q, k, v), "large scores")


def test_prefill_ignores_unwritten_cache_rows(ctx, oracle, forced):
    """Cache rows past pos + S hold NaN: no kernel may let them reach the output."""
    from test_gpu_attention import ref_attention_block
    rng = np.random.default_rng(21)
    S = 140
    kc_ref, vc_ref = np.zeros((32, 2048, 64), np.float16), np.zeros((32, 2048, 64), np.float16)
    poison = np.full((32, 2048, 64), np.nan, np.float16)
    kc, vc = ctx.upload(poison), ctx.upload(poison)
    qkv = f16_normal(rng, (S, 6144))
    ref = ref_attention_block(oracle, qkv, kc_ref, vc_ref, 0)
    out = ctx.alloc((S, 2048))
    ctx.sdpa_prefill_fused(ctx.upload(qkv), kc, vc, out, S, 32, 64, 2048, 0, 32)
    ctx.sync()
    got = out.numpy()
    assert np.isfinite(got.astype(np.float32)).all()
    assert_close_ref(got, ref, "prefill over a poisoned cache")


@pytest.mark.parametrize("crops", [1, 3, 13])
def test_vit_layout(ctx, oracle, forced, crops):
    """Heads interleaved inside the packed qkv rows (row stride 3456, head stride 72), one batch per crop."""
    rng = np.random.default_rng(crops + 40)
    T, H, d = 729, 16, 72
    qkv = f16_normal(rng, (crops * T, 3 * H * d))
    out = ctx.alloc((crops * T, H * d))
    ctx.sdpa_vit_fused(ctx.upload(qkv), out, crops, T, H, d)
    ctx.sync()
    got = out.numpy()
    for c in range(crops):
        blk = qkv[c * T:(c + 1) * T]
        q, k, v = [np.ascontiguousarray(blk[:, i * H * d:(i + 1) * H * d].reshape(T, H, d).transpose(1, 0, 2))
                   for i in range(3)]
        ref = np.ascontiguousarray(oracle.sdpa_maskless(q, k, v).transpose(1, 0, 2)).reshape(T, H * d)
        assert_close_ref(got[c * T:(c + 1) * T], ref, f"crop {c}")


_WALK: dict = {}


@pytest.mark.parametrize("per_sm", [0, 1, 2])
def test_ctas_that_walk_several_items_give_the_same_result(ctx, oracle, per_sm):
    """The tcgen05 kernel's grid is capped at attn_ctas_per_sm CTAs per SM; a CTA then walks several (query block,
    head, batch) items, carrying its rings, S / P buffers and wait parities from one item to the next.  13 crops are
    1248 items (4-9 per CTA); the causal case (320 items) has items of 2 to 20 key tiles in one CTA's walk.  per_sm = 0 gives
    every item its own CTA.  All three against the oracle, and bit-equal to one another."""
    ctx.set_option("attn_tc", 1)
    ctx.set_option("attn_ctas_per_sm", per_sm)
    try:
        rng = np.random.default_rng(77)
        crops, T, H, d = 13, 729, 16, 72
        qkv = f16_normal(rng, (crops * T, 3 * H * d))
        out = ctx.alloc((crops * T, H * d))
        ctx.sdpa_vit_fused(ctx.upload(qkv), out, crops, T, H, d)
        ctx.sync()
        got = out.numpy()
        for c in (0, 6, 12):
            blk = qkv[c * T:(c + 1) * T]
            q, k, v = [np.ascontiguousarray(blk[:, i * H * d:(i + 1) * H * d].reshape(T, H, d).transpose(1, 0, 2))
                       for i in range(3)]
            ref = np.ascontiguousarray(oracle.sdpa_maskless(q, k, v).transpose(1, 0, 2)).reshape(T, H * d)
            assert_close_ref(got[c * T:(c + 1) * T], ref, f"crop {c}")
        S = 1230
        qkv2 = f16_normal(rng, (S, 6144))
        kc, vc, o2 = ctx.alloc((32, 2048, 64)), ctx.alloc((32, 2048, 64)), ctx.alloc((S, 2048))
        ctx.sdpa_prefill_fused(ctx.upload(qkv2), kc, vc, o2, S, 32, 64, 2048, 0, 32)
        ctx.sync()
        got2 = o2.numpy()
    finally:
        ctx.set_option("attn_ctas_per_sm", 2)
        ctx.set_option("attn_tc", -1)
    _WALK[per_sm] = (got, got2)
    if per_sm == 0:   # the causal case against the oracle once; the other grids must equal this one bit for bit
        from test_gpu_attention import ref_attention_block
        kc_ref, vc_ref = np.zeros((32, 2048, 64), np.float16), np.zeros((32, 2048, 64), np.float16)
        assert_close_ref(got2, ref_attention_block(oracle, qkv2, kc_ref, vc_ref, 0), "causal prefill of 1230 rows")
    elif 0 in _WALK:
        np.testing.assert_array_equal(got, _WALK[0][0])
        np.testing.assert_array_equal(got2, _WALK[0][1])


_MASKED_WALK: dict = {}


@pytest.mark.parametrize("per_sm", [0, 1, 2])
def test_masked_ctas_that_walk_over_unseen_query_blocks(ctx, oracle, per_sm):
    """Masked items of one CTA's walk over different spans of keys: whole 128-row blocks that see nothing stand first, last, alone and
    three in a row.  56 heads of 12 blocks are 672 items, 4 or 5 per CTA (per_sm 1), 2 or 3 (per_sm 2) or one (per_sm 0).  They
    must not put the roles' barriers out of step: against the oracle, zeros where nothing is seen (the first keys, which only an
    unseen block's one tile visits, have infinite values), three launches in a row and all three grids bit for bit."""
    H, lq, lk = 56, 1500, 700
    rng = np.random.default_rng(31)
    q, k, v = f16_normal(rng, (H, lq, 64)), f16_normal(rng, (H, lk, 64)), f16_normal(rng, (H, lk, 64))
    m = (rng.random((lq, lk)) < 0.6).astype(np.uint8)
    for b in range(12):
        rows = m[b * 128:(b + 1) * 128]
        lo = 64 + (b * 61) % 450
        rows[:, :lo] = 0
        rows[:, lo + 90 + 20 * b:] = 0
        rows[:, lo] = 1
        if b in (0, 3, 4, 5, 8, 11):
            rows[:] = 0
    v[:, :64] = np.inf
    ctx.set_option("attn_tc", 1)
    ctx.set_option("attn_ctas_per_sm", per_sm)
    try:
        got = [ctx.sdpa_masked(q, k, v, m, H, lq, lk, 64) for _ in range(3)]
    finally:
        ctx.set_option("attn_ctas_per_sm", 2)
        ctx.set_option("attn_tc", -1)
    for again in got[1:]:
        np.testing.assert_array_equal(again, got[0])
    seen = m.any(1)
    assert (got[0][:, ~seen] == 0).all()
    if not _MASKED_WALK:
        _MASKED_WALK["ref"] = oracle.sdpa_masked(q, k[:, 64:].copy(), v[:, 64:].copy(), m[:, 64:].copy())[:, seen]
    assert_close_ref(got[0][:, seen], _MASKED_WALK["ref"], "unseen query blocks")
    np.testing.assert_array_equal(got[0], _MASKED_WALK.setdefault("first", got[0]))


def _masked_case(rng, h, lq, lk):
    q, k, v = f16_normal(rng, (h, lq, 64)), f16_normal(rng, (h, lk, 64)), f16_normal(rng, (h, lk, 64))
    m = (rng.random((lq, lk)) < 0.5).astype(np.uint8)
    m[:, 0] = 1
    return q, k, v, m


def _plain_edges(graph) -> bool:
    """Are all edges of a torch-captured graph full dependencies?  (This form of the query refuses edges with data.)"""
    n = C.c_size_t(64)
    ends = (C.c_void_p * 64)(), (C.c_void_p * 64)()
    status = C.CDLL("libcudart.so.12").cudaGraphGetEdges(C.c_void_p(int(graph.raw_cuda_graph())), *ends, C.byref(n))
    assert status != 0 or n.value > 2
    return status == 0


@pytest.mark.parametrize("owner", ["context", "stream"])
def test_masked_attention_in_a_captured_graph(pkg, oracle, owner):
    """The first calls of a context inside a capture, begun by md_graph_begin or by the owner of the stream the context was given (with
    the strictest capture mode): a product, and the masked attention with its temporary memory, on plain edges, replayed over changed inputs."""
    import torch
    rng = np.random.default_rng(4)
    h, lq, lk = 4, 200, 333
    ctx, stream = pkg.Context(0), torch.cuda.Stream()
    bufs = [torch.from_numpy(x).cuda() for x in _masked_case(rng, h, lq, lk)]
    a, w = torch.randn(16, 256, device="cuda").half(), torch.randn(512, 256, device="cuda").half()
    out, prod = torch.empty(h, lq, 64, dtype=torch.half, device="cuda"), torch.empty(16, 512, dtype=torch.half, device="cuda")
    ptr = [b.data_ptr() for b in bufs]
    ctx.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()

    def calls():
        ctx.hgemm_nt(a.data_ptr(), w.data_ptr(), 16, 512, 256, out=prod.data_ptr())
        ctx.sdpa_masked(*ptr, h, lq, lk, 64, out=out.data_ptr())
        ctx.sdpa_masked(*ptr, h, lq, lk, 64, out=out.data_ptr())

    if owner == "context":
        ctx.graph_begin()
        calls()
        g = ctx.graph_end()
        replay = lambda: ctx.graph_launch(g)
    else:
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=stream, capture_error_mode="global"):
            calls()
        assert _plain_edges(g)
        replay = g.replay
    for _ in range(3):
        case = _masked_case(rng, h, lq, lk)
        for b, x in zip(bufs, case):
            b.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            replay()
            replay()
        torch.cuda.synchronize()
        assert_close_ref(out.cpu().numpy(), oracle.sdpa_masked(*case), "replayed")
        assert_close_ref(prod.cpu().numpy(), (a.float() @ w.float().T).cpu().numpy(), "replayed product")
    if owner == "context":
        ctx.graph_destroy(g)
    else:
        del g, replay
    ctx.close()


def test_masked_attention_on_two_streams(pkg, oracle):
    """A context that is moved between two streams: each call's mask words are its own while both are in flight."""
    import torch
    rng = np.random.default_rng(6)
    ctx, streams = pkg.Context(0), [torch.cuda.Stream(), torch.cuda.Stream()]
    shapes = [(8, 700, 900), (8, 650, 1000)]
    cases = [_masked_case(rng, *s) for s in shapes]
    bufs = [[torch.from_numpy(x).cuda() for x in c] for c in cases]
    outs = [[torch.empty(s[0], s[1], 64, dtype=torch.half, device="cuda") for _ in range(6)] for s in shapes]
    torch.cuda.synchronize()
    for i in range(6):
        for s in (0, 1):
            ctx.set_stream(streams[s].cuda_stream)
            ctx.sdpa_masked(*[b.data_ptr() for b in bufs[s]], *shapes[s], 64, out=outs[s][i].data_ptr())
    torch.cuda.synchronize()
    for s in (0, 1):
        ref = oracle.sdpa_masked(*cases[s])
        for o in outs[s]:
            assert_close_ref(o.cpu().numpy(), ref, f"stream {s}")
    ctx.set_stream(None)
    ctx.close()


def test_masked_attention_when_no_device_memory_is_left(pkg, oracle):
    """A host may have taken all of the device's memory before it calls: the masked attention, which wants some for its mask's bits, then
    takes the kernel that reads the bytes."""
    rng = np.random.default_rng(8)
    h, lq, lk = 4, 200, 2100
    case = _masked_case(rng, h, lq, lk)
    ctx, taken = pkg.Context(0), []
    args = [ctx.upload(x) for x in case]
    out = ctx.alloc((h, lq, 64))
    ref = oracle.sdpa_masked(*case)
    small = [ctx.upload(x) for x in _masked_case(rng, h, 8, 64)]
    ctx.sdpa_masked(*small, h, 8, 64, 64, out=out)          # the kernel that reads bytes, loaded
    ctx.sync()
    size = 16 << 30
    while size >= 1 << 16 and len(taken) < 400:
        try:
            taken.append(ctx.alloc((size,), np.uint8))
        except pkg.MdError:
            size //= 4
    try:
        ctx.sdpa_masked(*args, h, lq, lk, 64, out=out)
        ctx.sync()
    finally:
        for b in taken:
            ctx.release(b)
    assert_close_ref(out.numpy(), ref, "no memory left")
    ctx.sdpa_masked(*args, h, lq, lk, 64, out=out)
    ctx.sync()
    assert_close_ref(out.numpy(), ref, "memory again")
    ctx.close()


def test_forced_tcgen05_rejects_other_head_dims(ctx, pkg):
    ctx.set_option("attn_tc", 1)
    try:
        z = np.zeros((2, 8, 48), np.float16)
        with pytest.raises(pkg.MdError):
            ctx.sdpa_maskless(z, z, z, 2, 8, 8, 48)
    finally:
        ctx.set_option("attn_tc", -1)
