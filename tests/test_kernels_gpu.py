"""Numerics of every CUDA kernel against the fp32 PyTorch statement of the same operator."""
import ctypes
import math

import pytest
import torch

from lorax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    from lorax_b200.ops import native
    native.load()
    return native


def _rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-6)).item()


@pytest.mark.parametrize("T,N,K", [(1, 512, 256), (7, 384, 512), (16, 4096, 4096), (33, 1024, 14336), (100, 6144, 4096),
                                   (128, 4096, 4096), (200, 1000, 520), (256, 2048, 1024)])
def test_gemm_small_t(nat, T, N, K):
    torch.manual_seed(T * 7 + N)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    out = nat.gemm(x, w)
    torch.cuda.synchronize()
    nat.workspace().check_status()
    want = x.float() @ w.float().t()
    assert _rel_err(out, want) < 6e-3
    # deterministic (split-K reduces in a fixed order)
    out2 = nat.gemm(x, w)
    assert torch.equal(out, out2)


@pytest.mark.parametrize("T,N,K", [(257, 512, 512), (1000, 4096, 4096), (4096, 6144, 4096), (300, 1000, 520)])
def test_gemm_large_t(nat, T, N, K):
    torch.manual_seed(T + N)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    b = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    out = nat.gemm(x, w, bias=b)
    torch.cuda.synchronize()
    nat.workspace().check_status()
    want = x.float() @ w.float().t() + b.float()
    assert _rel_err(out, want) < 6e-3


@pytest.mark.parametrize("mode", [1, 2])
def test_gemm_modes_bias_split(nat, mode):
    torch.manual_seed(3)
    T, N, K = 48, 640, 2048
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    b = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    want = x.float() @ w.float().t() + b.float()
    for split in ([1, 2, 4] if mode == 1 else [0]):
        out = nat.gemm(x, w, bias=b, mode=mode, force_split=split)
        torch.cuda.synchronize()
        nat.workspace().check_status()
        assert _rel_err(out, want) < 6e-3, (mode, split)


@pytest.mark.parametrize("T,N,K,bn", [(16, 4096, 4096, 0), (64, 28672, 4096, 0), (256, 6144, 4096, 64), (256, 4096, 14336, 256),
                                      (200, 1000, 520, 0), (576, 4096, 4096, 0), (700, 28672, 1024, 0), (1000, 4096, 14336, 0)])
def test_gemm_stream_k(nat, T, N, K, bn):
    """The partly filled last wave is cut along K across all SMs (policy 2 forces it); policy 1 computes whole tiles."""
    torch.manual_seed(T + N + K)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    b = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    want = x.float() @ w.float().t() + b.float()
    base = 1 if T <= 256 else 2
    outs = []
    for policy in (1, 2, 2):
        out = nat.gemm(x, w, bias=b, mode=base | (policy << 8), force_split=bn << 16)
        torch.cuda.synchronize()
        nat.workspace().check_status()
        assert _rel_err(out, want) < 6e-3, policy
        outs.append(out)
    assert torch.equal(outs[1], outs[2])          # fixed reduction order
    assert _rel_err(outs[1], outs[0]) < 2e-3


def test_gemm_strided_views(nat):
    torch.manual_seed(4)
    big = torch.randn(40, 3 * 1024, device="cuda", dtype=torch.bfloat16)
    x = big[:, 1024:2048]
    w = torch.randn(256, 1024, device="cuda", dtype=torch.bfloat16) / 32
    outbuf = torch.zeros(40, 512, device="cuda", dtype=torch.bfloat16)
    nat.gemm(x, w, out=outbuf[:, 256:])
    torch.cuda.synchronize()
    assert _rel_err(outbuf[:, 256:], x.float() @ w.float().t()) < 6e-3
    assert outbuf[:, :256].abs().max().item() == 0


@pytest.mark.parametrize("T,H,layernorm", [(5, 4096, False), (64, 8192, False), (3, 256, False), (9, 1024, True)])
def test_norm_residual(nat, T, H, layernorm):
    torch.manual_seed(0)
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    r = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(H, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(H, device="cuda", dtype=torch.bfloat16) if layernorm else None
    r_ref = r.clone()
    want = ref.norm_residual(x, r_ref, w, 1e-5, bias=b, layernorm=layernorm, weight_offset=1.0 if not layernorm else 0.0)
    got = nat.norm_residual(x, r, w, 1e-5, bias=b, layernorm=layernorm, weight_offset=1.0 if not layernorm else 0.0)
    assert torch.equal(r, r_ref)
    assert _rel_err(got, want) < 5e-3
    got2 = nat.norm_residual(x, None, w, 1e-5, bias=b, layernorm=layernorm)
    want2 = ref.norm_residual(x, None, w, 1e-5, bias=b, layernorm=layernorm)
    assert _rel_err(got2, want2) < 5e-3


@pytest.mark.parametrize("nh,nkv,d,rot", [(32, 8, 128, 128), (4, 2, 64, 64), (8, 8, 64, 32)])
def test_rope_kvwrite(nat, nh, nkv, d, rot):
    torch.manual_seed(1)
    T, page, blocks = 37, 32, 12
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32)
    cs = ref.rope_cache(rot, 512, 10000.0, device="cuda")
    slots = torch.randperm(blocks * page, device="cuda")[:T].to(torch.int32)
    slots[3] = -1
    cache = torch.zeros(blocks, nkv, 2, page, d, device="cuda", dtype=torch.bfloat16)
    cache_ref = cache.clone()
    qkv_ref = qkv.clone()
    ref.rope_kvwrite(qkv_ref, pos, cs, cache_ref, slots, nh, nkv, d, rot)
    nat.rope_kvwrite(qkv, pos, cs, cache, slots, nh, nkv, d, rot)
    assert _rel_err(qkv, qkv_ref) < 4e-3
    assert _rel_err(cache, cache_ref) < 4e-3


def test_prefill_metadata(nat):
    """Per-token positions, cache slots and adapter slots of a ragged prefill, computed on the device from the per-sequence arrays."""
    q_lens, cache_lens, slots_of = [5, 64, 1, 130, 33], [0, 7, 99, 32, 0], [-1, 3, 3, 0, -1]
    B, page, max_blocks = len(q_lens), 32, 9
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), device="cuda", dtype=torch.int32)
    cl = torch.tensor(cache_lens, device="cuda", dtype=torch.int32)
    ss = torch.tensor(slots_of, device="cuda", dtype=torch.int32)
    bt = torch.randint(1, 500, (B, max_blocks), device="cuda", dtype=torch.int32)
    T = sum(q_lens)
    got = nat.prefill_metadata(cu, cl, ss, bt, page, T)
    want = ref.prefill_metadata(cu, cl, ss, bt, page, T)
    for g, w in zip(got, want):
        assert torch.equal(g, w)
    # against the definition
    t = 5 + 64 + 1 + 17                     # token 17 of sequence 3
    assert int(got[0][t]) == 32 + 17 and int(got[1][t]) == int(bt[3, (32 + 17) // page]) * page + (32 + 17) % page and int(got[2][t]) == 0


@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_pytorch_tanh"])
def test_act_mul(nat, act):
    x = torch.randn(19, 2 * 1376, device="cuda", dtype=torch.bfloat16)
    assert _rel_err(nat.act_mul(x, 1376, act), ref.act_mul(x, 1376, act)) < 4e-3
    assert _rel_err(nat.act_mul(x, 1376, act, gated=False), ref.act_mul(x, 1376, act, gated=False)) < 4e-3


@pytest.mark.parametrize("T, V, ld", [(1, 32000, 32000), (1, 128256, 128256), (37, 32000, 32000), (38, 32000, 32000), (75, 32003, 32008), (149, 4096, 4096),
                                      (3, 50257, 50257), (2, 7, 8), (5, 4097, 4104)])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_argmax_logprob_over_split_rows(nat, T, V, ld, softcap):
    """Rows over clusters of one to eight CTAs, rows that start off a 16-byte boundary, ties across the parts, masked logits.  The sum of
    V terms in fp32 in any order is within V * 2^-24 of itself relatively, and so is its logarithm; expf and logf add a few 2^-22."""
    g = torch.Generator().manual_seed(V + T)
    logits = (torch.randn(T, ld, generator=g) * 3).to(torch.bfloat16)
    logits[0, : V // 3] = float("-inf")
    logits[T - 1, [V // 5, V - 1, V // 2]] = 40.0
    logits = logits.cuda()[:, :V]
    i, lp = nat.argmax_logprob(logits, softcap=softcap)
    x = logits.double()
    if softcap:
        x = softcap * torch.tanh(x / softcap)
    top = x.max(-1).values
    assert torch.equal(logits.gather(1, i.long()[:, None])[:, 0], logits.max(-1).values)
    assert torch.equal(i.cpu().long(), (logits == logits.max(-1, keepdim=True).values).int().argmax(-1).cpu())
    assert torch.allclose(lp.double(), top - torch.logsumexp(x, -1), atol=V * 2 ** -24 + 2 ** -18, rtol=2 ** -20)


@pytest.mark.parametrize("n", [1, 127, 129])
def test_place_rows(nat, n):
    g = torch.Generator().manual_seed(n)
    job = torch.stack([torch.randperm(200, generator=g)[:n]] + [torch.randint(0, 9999, (n,), generator=g) for _ in range(3)]).to(torch.int32)
    want = [torch.randint(0, 99, (200,), generator=g, dtype=torch.int32) for _ in range(4)]
    got = [t.clone().cuda() for t in want]
    ref.place_rows(job, *want)
    nat.place_rows(job.cuda(), *got)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)


def test_embed_argmax_advance(nat):
    table = torch.randn(1000, 256, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, 2000, (50,), device="cuda", dtype=torch.int32)
    got = nat.embed(ids, table, v0=500, v1=1500, mult=2.0)
    want = ref.embed(ids, table, v0=500, v1=1500, mult=2.0)
    assert torch.equal(got, want)
    logits = torch.randn(33, 32000, device="cuda", dtype=torch.bfloat16)
    i, lp = nat.argmax_logprob(logits)
    wi, wlp = ref.argmax_logprob(logits)
    assert torch.equal(i.long(), wi.long())
    assert torch.allclose(lp, wlp, atol=2e-3)
    B, page = 9, 32
    bt = torch.randint(1, 100, (B, 8), device="cuda", dtype=torch.int32)
    state = [torch.randint(0, 100, (B,), device="cuda", dtype=torch.int32) for _ in range(2)]
    inp, pos = state
    ctx = pos + 1
    ctx[2] = 0
    slots = torch.zeros(B, device="cuda", dtype=torch.int32)
    nxt = torch.randint(0, 100, (B,), device="cuda", dtype=torch.int32)
    a = [t.clone() for t in (inp, pos, ctx, slots)]
    b = [t.clone() for t in (inp, pos, ctx, slots)]
    nat.advance_decode(a[0], nxt, a[1], a[2], a[3], bt, page)
    ref.advance_decode(b[0], nxt, b[1], b[2], b[3], bt, page)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


def _make_cache(B, max_len, nkv, d, page=32, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    max_blocks = (max_len + page - 1) // page
    nblocks = B * max_blocks + 1
    cache = torch.randn(nblocks, nkv, 2, page, d, device="cuda", dtype=torch.bfloat16, generator=g)
    perm = torch.randperm(nblocks - 1, device="cuda", generator=g)[: B * max_blocks] + 1
    bt = perm.view(B, max_blocks).to(torch.int32)
    return cache, bt


@pytest.mark.parametrize("nh,nkv,d,window,softcap,nsplit", [(32, 8, 128, 0, 0.0, 1), (32, 8, 128, 100, 0.0, 1),
                                                             (4, 2, 64, 0, 0.0, 1), (8, 8, 128, 0, 30.0, 1),
                                                             (32, 8, 128, 0, 0.0, 4), (32, 1, 128, 0, 0.0, 2)])
def test_attn_decode(nat, nh, nkv, d, window, softcap, nsplit):
    torch.manual_seed(5)
    B, max_len = 11, 700
    cache, bt = _make_cache(B, max_len, nkv, d)
    ctx = torch.randint(1, max_len, (B,), device="cuda", dtype=torch.int32)
    ctx[0] = 1
    ctx[1] = max_len
    ctx[2] = 0
    q = torch.randn(B, nh * d, device="cuda", dtype=torch.bfloat16)
    scale = d ** -0.5
    got = nat.attn_decode(q, cache, bt, ctx, nh, nkv, d, scale, window, softcap, nsplit)
    want = ref.attn_decode(q, cache, bt, ctx, nh, nkv, d, scale, window, softcap)
    assert _rel_err(got, want) < 1e-2


@pytest.mark.parametrize("nh,nkv,d,window,cached", [(32, 8, 128, 0, False), (4, 2, 64, 0, True), (8, 2, 128, 70, True)])
def test_attn_prefill(nat, nh, nkv, d, window, cached):
    torch.manual_seed(6)
    q_lens = [5, 64, 130, 257, 1]
    B = len(q_lens)
    cache_lens = [0, 3, 64, 100, 31] if cached else [0] * B
    max_len = max(a + b for a, b in zip(q_lens, cache_lens))
    cache, bt = _make_cache(B, max_len, nkv, d, seed=1)
    T = sum(q_lens)
    q = torch.randn(T, nh * d, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), device="cuda", dtype=torch.int32)
    cl = torch.tensor(cache_lens, device="cuda", dtype=torch.int32)
    ts, tq = ref.prefill_tiles(q_lens)
    ts = torch.tensor(ts, device="cuda", dtype=torch.int32)
    tq = torch.tensor(tq, device="cuda", dtype=torch.int32)
    scale = d ** -0.5
    got = nat.attn_prefill(q, cache, bt, cu, cl, ts, tq, nh, nkv, d, scale, window)
    want = ref.attn_prefill(q, cache, bt, cu, cl, ts, tq, nh, nkv, d, scale, window)
    assert _rel_err(got, want) < 1e-2


@pytest.mark.parametrize("nh,nkv,d,rot", [(32, 8, 128, 128), (4, 2, 64, 32)])
def test_fp8_kv_cache(nat, nh, nkv, d, rot):
    """e4m3 KV pages with a K and a V scale: `rope_kvwrite` stores value / scale (saturating), decode and prefill attention read
    stored value * scale.  The bytes written match the fp32 reference bit for bit (up to the rounding of the rotated bf16 value),
    and attention over the same fp8 cache matches fp32 attention over its dequantised values; against the bf16 cache the error is
    the quantisation's."""
    torch.manual_seed(21)
    page, ks, vs = 32, 0.05, 0.02
    # ---- writes
    T, blocks = 41, 12
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device="cuda", dtype=torch.bfloat16) * 3
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32)
    cs = ref.rope_cache(rot, 512, 10000.0, device="cuda")
    slots = torch.randperm(blocks * page, device="cuda")[:T].to(torch.int32)
    slots[5] = -1
    cache = torch.zeros(blocks, nkv, 2, page, d, device="cuda", dtype=torch.float8_e4m3fn)
    cache_ref = torch.zeros_like(cache)
    qkv_ref = qkv.clone()
    ref.rope_kvwrite(qkv_ref, pos, cs, cache_ref, slots, nh, nkv, d, rot, kv_scale=(ks, vs))
    nat.rope_kvwrite(qkv, pos, cs, cache, slots, nh, nkv, d, rot, kv_scale=(ks, vs))
    a, b = cache.float(), cache_ref.float()
    assert (a != b).float().mean() < 0.02                  # a rotated value that rounds differently in bf16 may land one e4m3 step away
    assert _rel_err(a, b) < 2e-2
    assert a.abs().max() <= 448 and torch.isfinite(a).all()        # 3 * N(0,1) / 0.02 saturates instead of overflowing
    # ---- reads
    B, max_len = 9, 600
    wide, bt = _make_cache(B, max_len, nkv, d, seed=3)
    kq = torch.empty_like(wide, dtype=torch.float8_e4m3fn)
    kq.view(torch.uint8)[:, :, 0] = ref._to_e4m3_bytes(wide[:, :, 0], ks)
    kq.view(torch.uint8)[:, :, 1] = ref._to_e4m3_bytes(wide[:, :, 1], vs)
    ctx = torch.randint(1, max_len, (B,), device="cuda", dtype=torch.int32)
    ctx[0], ctx[1] = 1, max_len
    q = torch.randn(B, nh * d, device="cuda", dtype=torch.bfloat16)
    scale = d ** -0.5
    for nsplit in (1, 4):
        got = nat.attn_decode(q, kq, bt, ctx, nh, nkv, d, scale, 0, 0.0, nsplit, kv_scale=(ks, vs))
        want = ref.attn_decode(q, kq, bt, ctx, nh, nkv, d, scale, 0, 0.0, kv_scale=(ks, vs))
        assert _rel_err(got, want) < 1e-2, nsplit
    assert _rel_err(got, ref.attn_decode(q, wide, bt, ctx, nh, nkv, d, scale)) < 8e-2        # quantisation error only
    q_lens, cache_lens = [70, 200, 33], [0, 150, 64]
    Tq = sum(q_lens)
    qp = torch.randn(Tq, nh * d, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), device="cuda", dtype=torch.int32)
    cl = torch.tensor(cache_lens, device="cuda", dtype=torch.int32)
    ts, tq = ref.prefill_tiles(q_lens)
    ts, tq = torch.tensor(ts, device="cuda", dtype=torch.int32), torch.tensor(tq, device="cuda", dtype=torch.int32)
    got = nat.attn_prefill(qp, kq, bt[:3], cu, cl, ts, tq, nh, nkv, d, scale, 0, kv_scale=(ks, vs))
    want = ref.attn_prefill(qp, kq, bt[:3], cu, cl, ts, tq, nh, nkv, d, scale, 0, kv_scale=(ks, vs))
    assert _rel_err(got, want) < 1e-2
    nat.workspace().check_status()


@pytest.mark.parametrize("nh,nkv,window,softcap,q_lens,cache_lens", [
    (32, 8, 0, 0.0, [700, 1300, 3], [0, 0, 0]),                # several key blocks per tile: both TMEM buffers and both K/V stages cycle
    (8, 2, 0, 0.0, [200, 64, 129], [900, 37, 128]),            # chunks that continue a cached prefix (chunked prefill, prefix cache)
    (16, 4, 300, 0.0, [1000, 50], [0, 2000]),                  # sliding window: key blocks left of the window are skipped
    (8, 4, 0, 30.0, [333], [5])])                              # soft-capped scores
def test_attn_prefill_tensor_core(nat, nh, nkv, window, softcap, q_lens, cache_lens):
    """tcgen05 flash prefill (two heads of a KV group per CTA, K / V pages by TMA from the paged cache) against fp32 attention."""
    torch.manual_seed(16)
    d = 128
    assert nat.load().lx_attn_prefill_tc_supported(nh, nkv, d, nh * d, nh * d) == 1
    B = len(q_lens)
    max_len = max(a + b for a, b in zip(q_lens, cache_lens))
    cache, bt = _make_cache(B, max_len, nkv, d, seed=4)
    T = sum(q_lens)
    q = torch.randn(T, nh * d, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), device="cuda", dtype=torch.int32)
    cl = torch.tensor(cache_lens, device="cuda", dtype=torch.int32)
    ts, tq = ref.prefill_tiles(q_lens)
    ts = torch.tensor(ts, device="cuda", dtype=torch.int32)
    tq = torch.tensor(tq, device="cuda", dtype=torch.int32)
    scale = d ** -0.5
    for _ in range(2):
        got = nat.attn_prefill(q, cache, bt, cu, cl, ts, tq, nh, nkv, d, scale, window, softcap)
        torch.cuda.synchronize()
        nat.workspace().check_status()
        want = ref.attn_prefill(q, cache, bt, cu, cl, ts, tq, nh, nkv, d, scale, window, softcap)
        assert _rel_err(got, want) < 1e-2
        assert torch.isfinite(got.float()).all()


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("nh,nkv,window,softcap,bias,q_lens,cache_lens", [
    (8, 1, 0, 0.0, False, [1, 63, 64, 65], [0, 0, 127, 128]),      # two tiles a CTA; queries and keys around the edges of tiles and blocks
    (12, 2, 0, 0.0, False, [129, 192], [1, 300]),                  # six heads a group: one tile a CTA
    (4, 1, 1, 0.0, False, [130], [0]), (16, 4, 33, 0.0, False, [200, 5], [31, 700]), (4, 2, 128, 0.0, False, [257], [0]),
    (8, 2, 100, 20.0, False, [190, 66], [0, 250]), (8, 2, 0, 0.0, True, [150, 33], [0, 96]), (4, 2, 40, 15.0, True, [140], [64])])
def test_attn_prefill_tensor_core_tiles_and_masks(nat, nh, nkv, window, softcap, bias, q_lens, cache_lens, wide):
    """Every form of the scores and of their mask, with one and two tiles a CTA.  Weights are rounded to bf16 unless `wide`, results always:
    2^-9 each at most, relatively."""
    d, B, T = 128, len(q_lens), sum(q_lens)
    cache, bt = _make_cache(B, max(a + b for a, b in zip(q_lens, cache_lens)), nkv, d, seed=nh)
    q = torch.randn(T, nh * d, generator=torch.Generator("cuda").manual_seed(T), device="cuda").to(torch.bfloat16)
    ints = lambda v: torch.tensor(v, device="cuda", dtype=torch.int32)
    cu, cl = ints([0] + list(torch.tensor(q_lens).cumsum(0))), ints(cache_lens)
    ts, tq = (ints(t) for t in ref.prefill_tiles(q_lens))
    slopes = torch.linspace(0.01, 0.3, nh, device="cuda") if bias else None
    out, p, scale = torch.empty_like(q), nat._ptr, d ** -0.5
    rc = nat.load().lx_attn_prefill_tc(p(q), q.stride(0), T, p(cache), cache.shape[0], p(bt), bt.shape[1], p(cu), p(cl), p(ts), p(tq), ts.shape[0], p(out),
                                       out.stride(0), nh, nkv, d, window, scale, softcap, p(slopes), wide, p(nat.workspace().status), nat._stream())
    assert rc == 0
    nat.workspace().check_status()
    at = 0
    for b in range(B):
        n, m = q_lens[b], q_lens[b] + cache_lens[b]
        pos, key = cache_lens[b] + torch.arange(n, device="cuda")[:, None], torch.arange(m, device="cuda")
        for h in range(nh):
            k, v = cache[bt[b].long()][:, h * nkv // nh].transpose(0, 1).reshape(2, -1, d)[:, :m].double()
            s = q[at: at + n, h * d: (h + 1) * d].double() @ k.t() * scale
            s = softcap * torch.tanh(s / softcap) if softcap else s
            s = s + slopes[h].double() * key if bias else s
            s = s.masked_fill((key > pos) | ((pos - key >= window) if window else (key < 0)), float("-inf"))
            assert _rel_err(out[at: at + n, h * d: (h + 1) * d], torch.softmax(s, -1) @ v) < (2 ** -9 if wide else 2 ** -8)
        at += n


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("nh,nkv,window,softcap,bias", [(32, 8, 0, 0.0, False), (32, 8, 100, 0.0, False), (32, 8, 0, 20.0, False), (32, 8, 60, 20.0, False),
                                                        (32, 8, 0, 0.0, True), (32, 4, 200, 15.0, True),
                                                        (32, 16, 0, 0.0, False), (24, 4, 0, 20.0, False), (12, 2, 300, 20.0, False), (32, 16, 0, 0.0, True)])
def test_attn_prefill_tensor_core_of_many_tiles(nat, nh, nkv, window, softcap, bias, wide):
    """More tiles than SMs: two a CTA where a group has four heads or eight, one with two buffers of scores where it has two or six; one to eleven
    blocks of keys, blocks that all rows see whole among them."""
    test_attn_prefill_tensor_core_tiles_and_masks(nat, nh, nkv, window, softcap, bias, [1, 63, 64, 65, 129, 300, 40, 513], [0, 0, 127, 128, 300, 31, 1000, 900], wide)


def _by_blocks(q, k, v, first, scale, block=128):
    """Attention of one head in float64 the way prompt attention forms it: keys in blocks, weights rounded to bf16 relative to the largest
    score up to and including their block, divided by the sum of the unrounded weights.  q [n, d] at positions first .., k and v [m, d]."""
    t = q.double() @ k.double().t() * (scale * math.log2(math.e))
    t = t.masked_fill(torch.arange(k.shape[0], device=t.device) > first + torch.arange(q.shape[0], device=t.device)[:, None], float("-inf"))
    m = torch.full((q.shape[0], 1), float("-inf"), dtype=torch.float64, device=t.device)
    total = torch.zeros_like(m)
    o = torch.zeros(q.shape[0], v.shape[1], dtype=torch.float64, device=t.device)
    for kb in range(0, k.shape[0], block):
        s = t[:, kb: kb + block]
        top = torch.maximum(m, s.max(-1, keepdim=True).values)
        back, w = torch.exp2(m - top), torch.exp2(s - top)
        total = total * back + w.sum(-1, keepdim=True)
        o = o * back + w.to(torch.bfloat16).double() @ v[kb: kb + block].double()
        m = top
    return o / total


@pytest.mark.parametrize("q_lens,cache_lens,climb", [([137], [0], 0.0), ([700, 64], [0, 331], 0.0), ([500], [0], 0.012), ([300], [450], -0.012)])
def test_attn_prefill_weights_are_relative_to_the_largest_so_far(nat, q_lens, cache_lens, climb):
    """The rounding of prompt attention's weights, also where the scores climb or fall by `climb` (log2) from key to key: a near tie that a
    later layer decides on the last bits (the choice of an expert) comes out as before.  Only sums in fp32 and exp2 separate the kernel from the
    same in 64 bits: 2^-20 of sums that are up to 2^4 times the result, so that one bf16 word in a hundred rounds the other way, and a few
    weights in ten thousand.  (Weights relative to anything else are rounded otherwise: a tenth of all words differ and more.)"""
    nh, nkv, d = 8, 2, 128
    B, max_len = len(q_lens), max(a + b for a, b in zip(q_lens, cache_lens))
    cache, bt = _make_cache(B, max_len, nkv, d, seed=len(q_lens))
    g = torch.Generator().manual_seed(max_len)
    T = sum(q_lens)
    q = torch.randn(T, nh * d, generator=g).to(torch.bfloat16)
    q.view(T, nh, d)[:, :, 0] = 8.0
    q = q.cuda()
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), device="cuda", dtype=torch.int32)
    ts, tq = ref.prefill_tiles(q_lens)
    scale = d ** -0.5
    for b in range(B):
        n = -(-max_len // 32)
        rise = torch.arange(n * 32, device="cuda").view(n, 1, 32) * (climb / (8.0 * scale * math.log2(math.e)))
        cache[bt[b].long(), :, 0, :, 0] = rise.to(torch.bfloat16)
    got = nat.attn_prefill(q, cache, bt, cu, torch.tensor(cache_lens, device="cuda", dtype=torch.int32), torch.tensor(ts, device="cuda", dtype=torch.int32),
                           torch.tensor(tq, device="cuda", dtype=torch.int32), nh, nkv, d, scale)
    nat.workspace().check_status()
    at = 0
    for b in range(B):
        n, m = q_lens[b], q_lens[b] + cache_lens[b]
        pages = cache[bt[b].long()]                                            # [pages, nkv, 2, 32, d]
        for h in range(nh):
            kv = pages[:, h * nkv // nh].transpose(0, 1).reshape(2, -1, d)[:, :m]
            want = _by_blocks(q[at: at + n, h * d: (h + 1) * d], kv[0], kv[1], cache_lens[b], scale).to(torch.bfloat16)
            assert (got[at: at + n, h * d: (h + 1) * d] != want).float().mean() < 0.05, (b, h)
        at += n


@pytest.mark.parametrize("climb,softcap,window,cached", [(0.0, 0.0, 0, 0), (0.02, 0.0, 0, 300), (1.5, 0.0, 0, 0), (-0.3, 0.0, 0, 70), (0.4, 60.0, 200, 0)])
def test_attn_prefill_wide_weights_under_moving_maxima(nat, climb, softcap, window, cached):
    """Softmax weights of two bf16 terms where the largest score grows or falls by `climb` (log2) from key to key: from block to block the sums
    are rescaled by up to 2^192.  What remains is the rounding of the result: 2^-9 at most, 2^-9 / sqrt(3) = 1.1e-3 over all for evenly spread
    mantissas, up to 1.7e-3 where they gather above a power of two; the weights' two terms add 2^-17."""
    nh, nkv, d, n = 4, 2, 128, 700
    m = n + cached
    cache, bt = _make_cache(1, m, nkv, d, seed=n)
    scale = d ** -0.5
    pages = bt.shape[1]
    rise = torch.arange(pages * 32, device="cuda").view(pages, 1, 32) * (climb / (8.0 * scale * math.log2(math.e)))
    cache[bt[0].long(), :, 0, :, 0] = rise.to(torch.bfloat16)
    q = torch.randn(n, nh * d, device="cuda", dtype=torch.bfloat16)
    q.view(n, nh, d)[:, :, 0] = 8.0
    ints = lambda *v: torch.tensor(v, device="cuda", dtype=torch.int32)
    ts, tq = (ints(*t) for t in ref.prefill_tiles([n]))
    cu, cl, out, p = ints(0, n), ints(cached), torch.empty_like(q), nat._ptr
    rc = nat.load().lx_attn_prefill_tc(p(q), q.stride(0), n, p(cache), cache.shape[0], p(bt), bt.shape[1], p(cu), p(cl), p(ts), p(tq), ts.shape[0], p(out),
                                       out.stride(0), nh, nkv, d, window, scale, softcap, None, 1, p(nat.workspace().status), nat._stream())
    assert rc == 0
    nat.workspace().check_status()
    at = cached + torch.arange(n, device="cuda")[:, None]
    key = torch.arange(m, device="cuda")
    for h in range(nh):
        k, v = cache[bt[0].long()][:, h * nkv // nh].transpose(0, 1).reshape(2, -1, d)[:, :m].double()
        s = q[:, h * d: (h + 1) * d].double() @ k.t() * scale
        s = softcap * torch.tanh(s / softcap) if softcap else s
        s = s.masked_fill((key > at) | ((at - key >= window) if window else (key < 0)), float("-inf"))
        assert _rel_err(out[:, h * d: (h + 1) * d], torch.softmax(s, -1) @ v) < 1.8e-3


@pytest.mark.parametrize("B,nh,nkv,d,window,softcap,nsplit", [(5, 8, 8, 128, 0, 0.0, 1), (3, 32, 8, 128, 50, 0.0, 8), (40, 32, 8, 128, 0, 20.0, 4),
                                                            (6, 20, 1, 64, 0, 0.0, 2), (38, 16, 8, 64, 33, 0.0, 1), (2, 34, 2, 128, 0, 0.0, 1)])
def test_attn_decode_fp8_pages(nat, B, nh, nkv, d, window, softcap, nsplit):
    """Contexts around the edges of pages and of splits, groups of one to twenty heads, both CTA sizes, query rows that start on any 4-byte
    boundary and of any magnitude.  Weights and results are rounded to bf16 (2^-9 each, relatively)."""
    max_len = 700
    wide, bt = _make_cache(B, max_len, nkv, d, seed=B + d)
    cache = wide.to(torch.float8_e4m3fn)
    ctx = torch.randint(1, max_len, (B,), device="cuda", dtype=torch.int32)
    ctx[:2] = torch.tensor([1, 32])
    ctx[-1] = 33 if B > 2 else 64
    ldq = nh * d + 6
    q = torch.randn(B, ldq, device="cuda", dtype=torch.bfloat16)[:, 2: 2 + nh * d]
    q[0] *= 2.0 ** 20
    q[1] *= 2.0 ** -60
    q[-1, ::7] *= 2.0 ** -20
    got = nat.attn_decode(q, cache, bt, ctx, nh, nkv, d, d ** -0.5, window, softcap, nsplit, kv_scale=(0.5, 0.25))
    want = ref.attn_decode(q, cache, bt, ctx, nh, nkv, d, d ** -0.5, window, softcap, kv_scale=(0.5, 0.25))
    assert torch.isfinite(got).all()
    for b in range(B):
        assert _rel_err(got[b], want[b]) < 6e-3, (b, int(ctx[b]))


@pytest.mark.parametrize("nsplit,d", [(1, 128), (4, 128), (1, 64)])
def test_attn_decode_fp8_pages_keep_what_is_faint(nat, nsplit, d):
    """One key that takes nearly all of a row's weight, its value zero, beside 8000 of 2^-26 of it; and query rows whose largest element, 2^24
    times the others, meets zeros in every key.  The result hangs on what f16 loses without a scale.  Weights and results are rounded to 8
    bits at least, 2^-9 relatively, as over bf16 pages; the scores' sums in fp32 add 2^-22 of the scores (up to 20)."""
    nh, nkv, B, ctx = 8, 2, 3, 8001
    wide, bt = _make_cache(B, ctx, nkv, d, seed=d + nsplit)
    wide[:, :, 0] = 0.0
    wide[:, :, 1] = wide[:, :, 1].abs()
    q = torch.zeros(B, nh * d, device="cuda", dtype=torch.bfloat16)
    scale = d ** -0.5
    for b, at in ((0, 0), (1, 5000)):                                          # before and between the faint ones
        page = bt[b, at // 32].long()
        wide[page, :, 0, at % 32, 0] = round(18.3 / (8 * scale))
        wide[page, :, 1, at % 32] = 0.0
        q.view(B, nh, d)[b, :, 0] = 8.0
    wide[bt[2].long(), :, 0] = torch.randn_like(wide[bt[2].long(), :, 0])
    wide[bt[2].long(), :, 0, :, 0] = 0.0
    q[2] = torch.randn(nh * d, device="cuda") * 2
    q.view(B, nh, d)[2, :, 0] = 2.0 ** 24
    cache = wide.to(torch.float8_e4m3fn)
    lens = torch.full((B,), ctx, device="cuda", dtype=torch.int32)
    got = nat.attn_decode(q, cache, bt, lens, nh, nkv, d, scale, 0, 0.0, nsplit, kv_scale=(1.0, 0.5))
    for b in range(B):
        pages = cache[bt[b].long()].double()
        for h in range(nh):
            k, v = pages[:, h * nkv // nh].transpose(0, 1).reshape(2, -1, d)[:, :ctx]
            want = torch.softmax(q[b, h * d: (h + 1) * d].double() @ k.t() * scale, -1) @ v * 0.5
            assert want.abs().min() > 0 and _rel_err(got[b, h * d: (h + 1) * d], want) < 6e-3, (b, h)


@pytest.mark.parametrize("T, K", [(1, 4096), (7, 64), (9, 1000), (40, 14336), (33, 2056), (300, 512)])
def test_lora_shrink_short_steps(nat, T, K):
    """Clusters of one to eight CTAs over K, K off the blocks of 32, one and four row groups, ranks of 8 to 64, rows past the batch, dead entries.
    bf16 products are exact in fp32; a sum of K terms in fp32 is within K * 2^-24 of the sum of their magnitudes."""
    g = torch.Generator().manual_seed(T + K)
    ranks, nparts = [8, 16, 64, 32], 3
    bases, off = [], 0
    for r in ranks:
        bases.append(off)
        off += (r * (nparts * K + 8) + 63) // 64 * 64
    arena = (torch.randn(off, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(T, K + 8, generator=g).to(torch.bfloat16)
    tl, row = [], 0
    while row < T:
        n = min([3, 32, 8, 9, 17][len(tl) % 5], T - row)
        tl.append((len(tl) % 4, row, n, 0))
        row += n + len(tl) % 2
    tl[-1] = (tl[-1][0], tl[-1][1], 32, 0)                             # a table may be older than the batch
    table = torch.tensor(tl + [(-1, 0, 0, 0)] * 3, dtype=torch.int32)
    nat.workspace().lora_v.fill_(7.0)
    v = nat.lora_shrink_mma(x.cuda()[:, :K], table.cuda(), len(table), arena.cuda(), torch.tensor(bases).cuda(),
                            torch.tensor(ranks, dtype=torch.int32).cuda(), 0, nparts, 64, live_tiles=len(tl))
    nat.workspace().check_status()
    v = v[:T].cpu()
    seen = torch.zeros(T, v.shape[1], dtype=torch.bool)
    for slot, r0, n, _ in tl:
        n, R = min(n, T - r0), ranks[slot] * nparts
        A = arena[bases[slot]: bases[slot] + R * K].view(R, K).double()
        xs = x[r0: r0 + n, :K].double()
        assert ((v[r0: r0 + n, :R].double() - xs @ A.t()).abs() <= (xs.abs() @ A.abs().t()) * K * 2 ** -24 + 1e-30).all()
        seen[r0: r0 + n, :R] = True
    assert (v[~seen] == 7.0).all()


def _after_a_kernel(nat, product, T, K, rounds=6):
    """`product(x)` over inputs that a kernel which lets its successor start early has written directly in front: different ones in turn through
    one buffer, without a synchronisation in between.  -> the outputs, and the inputs they belong to."""
    srcs = [torch.randn(T, 2 * K, device="cuda", dtype=torch.bfloat16) * (1 + i) for i in range(2)]
    x = torch.zeros(T, K, device="cuda", dtype=torch.bfloat16)
    outs = []
    for i in range(rounds):
        nat.act_mul(srcs[i % 2], K, "silu", out=x)
        outs.append(product(x))
    torch.cuda.synchronize()
    return outs, [nat.act_mul(s, K, "silu") for s in srcs]


@pytest.mark.parametrize("T,N,K,mode,split", [
    (1, 4096, 4096, 0, 0), (13, 6144, 4096, 0, 0), (32, 4096, 14336, 0, 0),                # parts of K: a CTA's first block is not block 0
    (32, 512, 64, 0, 0), (33, 1024, 448, 0, 0), (33, 1024, 512, 0, 0), (33, 1000, 520, 0, 0),      # one, seven, eight and nine blocks in a ring of eight
    (129, 2048, 1024, 0, 0), (200, 1024, 256, 1, 0), (512, 1536, 1024, 2, 0), (300, 4096, 192, 2, 0),      # both orientations, rings of four and six
    (16, 1024, 4096, 1, 3), (64, 4096, 4096, 1 | 2 << 8, 0), (512, 6144, 2048, 2 | 2 << 8, 0), (513, 1024, 512, 0, 0)])
def test_gemm_reads_constant_weights_early(nat, T, N, K, mode, split):
    """Weights loaded in front of the wait: the same bits as behind it, however the product is cut."""
    torch.manual_seed(T + N)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    b = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    outs, xs = _after_a_kernel(nat, lambda x: nat.gemm(x, w, bias=b, mode=mode, force_split=split, w_const=True), T, K)
    want = [nat.gemm(x, w, bias=b, mode=mode, force_split=split) for x in xs]
    assert all(torch.equal(o, want[i % 2]) for i, o in enumerate(outs))
    assert _rel_err(want[1], xs[1].float() @ w.float().t() + b.float()) < 5e-3
    nat.workspace().check_status()


@pytest.mark.parametrize("between", ["norm", "act", "rope", "attention"])
@pytest.mark.parametrize("T,N,K", [(3, 4096, 1024), (64, 2048, 4096), (300, 1024, 512)])
def test_constant_weights_come_from_two_kernels_in_front(nat, T, N, K, between):
    """A kernel that lets its successor start early writes a product's weights, a short one that does not touch them stands in between: the
    one in front of the product does not write them, so it may say that they are constant."""
    torch.manual_seed(T + N)
    srcs = [torch.randn(N, 2 * K, device="cuda", dtype=torch.bfloat16) * (1 + i) for i in range(2)]
    w, x = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16), torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    small, ones = torch.randn(4, 1024, device="cuda", dtype=torch.bfloat16), torch.ones(1024, device="cuda", dtype=torch.bfloat16)
    cache, bt = _make_cache(4, 64, 2, 128)
    ints = lambda *v: torch.tensor(v, device="cuda", dtype=torch.int32)
    pos, slots, ctx, cos = ints(0, 1, 2, 3), ints(-1, -1, -1, -1), ints(5, 33, 64, 1), torch.rand(8, 128, device="cuda")
    step = dict(norm=lambda: nat.norm_residual(small, None, ones, 1e-5), act=lambda: nat.act_mul(small, 512),
                rope=lambda: nat.rope_kvwrite(small, pos, cos, cache, slots, 4, 2, 128, 128),
                attention=lambda: nat.attn_decode(small, cache, bt, ctx, 4, 2, 128, 0.1))[between]
    outs = []
    for i in range(6):
        nat.act_mul(srcs[i % 2], K, "silu", out=w)
        step()
        outs.append(nat.gemm(x, w, w_const=True))
    torch.cuda.synchronize()
    nat.workspace().check_status()
    want = [nat.gemm(x, nat.act_mul(s, K, "silu")) for s in srcs]
    assert all(torch.equal(o, want[i % 2]) for i, o in enumerate(outs))


@pytest.mark.parametrize("T,N,K,group", [(1, 4096, 1024, 128), (5, 28672, 4096, 128), (8, 8192, 384, 64), (9, 512, 2048, 128), (17, 1024, 256, 32), (32, 256, 128, 128)])
def test_packed_products_read_constant_codes_early(nat, T, N, K, group):
    from lorax_b200.utils.quant_formats import quantize_rtn
    torch.manual_seed(T + N)
    q = quantize_rtn(torch.randn(N, K, device="cuda") / math.sqrt(K), 4, group)
    outs, xs = _after_a_kernel(nat, lambda x: nat.gemm_wq(x, q, w_const=True), T, K)
    want = [nat.gemm_wq(x, q) for x in xs]
    assert all(torch.equal(o, want[i % 2]) for i, o in enumerate(outs))


@pytest.mark.parametrize("T,N,K", [(1, 512, 1024), (5, 640, 4096), (33, 1024, 384), (100, 256, 128), (300, 512, 1024)])
def test_fp8_products_read_weights_early(nat, T, N, K):
    torch.manual_seed(T + N)
    wq, sw = ref.quantize_weight_fp8_block128(torch.randn(N, K, device="cuda") / math.sqrt(K))
    outs, xs = _after_a_kernel(nat, lambda x: nat.gemm_fp8(x, wq, sw), T, K)
    want = []
    for x in xs:
        want.append(nat.gemm_fp8(x, wq, sw))
        torch.cuda.synchronize()
    assert all(torch.equal(o, want[i % 2]) for i, o in enumerate(outs))


@pytest.mark.parametrize("T", [7, 200])
def test_adapter_tables_of_the_kernel_in_front(nat, T):
    """Without `tables_const` table and ranks may come from the kernel directly in front, one that lets its successor start early; with it, and
    tables that lie there, the bits are the same."""
    g = torch.Generator().manual_seed(T)
    K, N, ranks, nparts = 1024, 1024, [16, 32, 48, 64], 2
    bases, off = [], 0
    for r in ranks:
        bases.append(off)
        off += r * (nparts * K + N)
    arena = (torch.randn(off, generator=g) * 0.05).to(torch.bfloat16).cuda()
    base = torch.tensor(bases).cuda()
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(N, K, generator=g) / 32).to(torch.bfloat16).cuda()
    G = 5
    host = torch.zeros(len(ranks) * 2 * G * 128, dtype=torch.uint8).pin_memory()
    for s, r in enumerate(ranks):
        nat.lora_encode_tmap(host[s * 2 * G * 128:], arena.data_ptr() + bases[s] * 2, K, nparts * r, r * (nparts * K + N), 1)
        nat.lora_encode_tmap_b(host[(s * 2 * G + G) * 128:], arena.data_ptr() + (bases[s] + r * nparts * K) * 2, r, N, r * (nparts * K + N), 1)
    maps = host.cuda()
    tables = [torch.tensor(ref.build_lora_tiles([(t // 5 + i) % 4 for t in range(T)], 32), dtype=torch.int32) for i in range(2)]
    n = tables[0].numel()
    assert tables[1].numel() == n and not torch.equal(*tables)
    size = max(n, 4)
    ints = [torch.zeros(size, device="cuda", dtype=torch.int32) for _ in range(4)]
    jobs = [torch.stack([torch.arange(n), t.flatten().long(), torch.tensor((ranks * n)[:n]), torch.zeros(n, dtype=torch.long)]).to(torch.int32).cuda() for t in tables]

    def passes(write):
        outs = []
        for i in range(6):
            table, rank = (ints[0][:n].view(-1, 4), ints[1][:4]) if write else (tables[i % 2].cuda(), torch.tensor(ranks, dtype=torch.int32).cuda())
            place = (lambda: nat.place_rows(jobs[i % 2], *ints)) if write else (lambda: torch.cuda.synchronize())
            known = dict(tables_const=not write)
            place()
            v = nat.lora_shrink_mma(x, table, len(table), arena, base, rank, 0, nparts, 64, **known)[:T].clone()
            y = torch.zeros(T, N, device="cuda", dtype=torch.bfloat16)
            v2 = v.nan_to_num(0.0)
            place()
            nat.lora_expand_tiles(v2, table, len(table), 32, arena, base, rank, nparts * K, y, N // 2, N, **known)
            place()
            z = nat.gemm_lora_fused(x, w, nat.LoraFused(table, len(table), len(table), maps, 2 * G, 0, G, rank, base, nparts, N // 2, N, 0, 64, arena, 0,
                                                        nparts * K, **known))
            outs.append((v, y, z))
        torch.cuda.synchronize()
        return outs

    nat.place_rows(jobs[1], *ints)
    torch.cuda.synchronize()
    nat.workspace().lora_v.zero_()
    want = passes(False)
    nat.workspace().lora_v.zero_()
    got = passes(True)
    nat.workspace().check_status()
    for a, b in zip(got, want):
        assert all(torch.equal(p, q) for p, q in zip(a, b))
        assert a[1].abs().sum() > 0


@pytest.mark.parametrize("nh,nkv,d,nsplit", [(12, 12, 64, 1), (32, 8, 128, 3), (6, 6, 128, 1)])
def test_attn_alibi(nat, nh, nkv, d, nsplit):
    """ALiBi slopes in both attention kernels (BLOOM, MPT): bias -slope_h * (query position - key position)."""
    from lorax_b200.models.decoder import alibi_slopes
    torch.manual_seed(15)
    slopes = alibi_slopes(nh).cuda()
    scale = d ** -0.5
    B, max_len = 7, 500
    cache, bt = _make_cache(B, max_len, nkv, d, seed=2)
    ctx = torch.randint(1, max_len, (B,), device="cuda", dtype=torch.int32)
    ctx[0], ctx[1] = 1, max_len
    q = torch.randn(B, nh * d, device="cuda", dtype=torch.bfloat16)
    got = nat.attn_decode(q, cache, bt, ctx, nh, nkv, d, scale, 0, 0.0, nsplit, alibi=slopes)
    want = ref.attn_decode(q, cache, bt, ctx, nh, nkv, d, scale, alibi=slopes)
    plain = ref.attn_decode(q, cache, bt, ctx, nh, nkv, d, scale)
    assert _rel_err(got, want) < 1e-2 and _rel_err(plain, want) > 0.1
    q_lens, cache_lens = [9, 150, 64], [0, 70, 33]
    cache, bt = _make_cache(3, 256, nkv, d, seed=3)
    T = sum(q_lens)
    q = torch.randn(T, nh * d, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), device="cuda", dtype=torch.int32)
    cl = torch.tensor(cache_lens, device="cuda", dtype=torch.int32)
    ts, tq = ref.prefill_tiles(q_lens)
    ts = torch.tensor(ts, device="cuda", dtype=torch.int32)
    tq = torch.tensor(tq, device="cuda", dtype=torch.int32)
    got = nat.attn_prefill(q, cache, bt, cu, cl, ts, tq, nh, nkv, d, scale, alibi=slopes)
    want = ref.attn_prefill(q, cache, bt, cu, cl, ts, tq, nh, nkv, d, scale, alibi=slopes)
    assert _rel_err(got, want) < 1e-2


@pytest.mark.parametrize("T", [3, 100, 700])
def test_lora_shrink_expand(nat, T):
    torch.manual_seed(8)
    K, parts = 1024, [512, 128, 128]
    N = sum(parts)
    ranks = [8, 16, 64, 32]
    unit_a, unit_b = 0, 3 * K        # per-unit-rank offsets of A_cat and B_cat inside a blob
    unit_total = 3 * K + N
    bases, off = [], 0
    for r in ranks:
        bases.append(off)
        off += r * unit_total
    arena = (torch.randn(off, device="cuda") * 0.05).to(torch.bfloat16)
    slot_base = torch.tensor(bases + [-1], device="cuda", dtype=torch.int64)
    slot_rank = torch.tensor(ranks + [0], device="cuda", dtype=torch.int32)
    # runs of equal slots plus base-model tokens
    tok_slot = torch.randint(-1, len(ranks), (T,), device="cuda", dtype=torch.int32)
    if T > 64:
        tok_slot = tok_slot[torch.arange(T, device="cuda") // 37 % tok_slot.numel()].contiguous()
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    v = torch.zeros(T, 3 * 64, device="cuda", dtype=torch.float32)
    v_ref = v.clone()
    nat.lora_shrink(x, tok_slot, arena, slot_base, slot_rank, unit_a, 3, 64, v)
    ref.lora_shrink(x, tok_slot, arena, slot_base, slot_rank, unit_a, 3, 64, v_ref)
    torch.cuda.synchronize()
    assert _rel_err(v, v_ref) < 2e-3
    y = torch.randn(T, N, device="cuda", dtype=torch.bfloat16)
    y_ref = y.clone()
    nat.lora_expand(v_ref, tok_slot, arena, slot_base, slot_rank, unit_b, y, parts[0], parts[0] + parts[1])
    ref.lora_expand(v_ref, tok_slot, arena, slot_base, slot_rank, unit_b, y_ref, parts[0], parts[0] + parts[1])
    nat.workspace().check_status()
    assert _rel_err(y, y_ref) < 5e-3


@pytest.mark.parametrize("T,max_rows", [(40, 32), (300, 32), (700, 128)])
def test_lora_tiled_tensor_core(nat, T, max_rows):
    """Tile-table LoRA: tcgen05 shrink through per-slot tensor maps + tiled expand, against the PyTorch loop."""
    torch.manual_seed(9)
    K, parts, L = 1024, [512, 128, 128], 3
    N = sum(parts)
    ranks = [8, 16, 64, 32]
    layer_units = 3 * K + N                    # A_cat (3 parts) then B_cat, per unit rank
    bases, off = [], 0
    for r in ranks:
        bases.append(off)
        off += r * layer_units * L
        off = (off + 63) // 64 * 64
    arena = (torch.randn(off, device="cuda") * 0.05).to(torch.bfloat16)
    slot_base = torch.tensor(bases, device="cuda", dtype=torch.int64)
    slot_rank = torch.tensor(ranks, device="cuda", dtype=torch.int32)
    G = 5
    tm_host = torch.zeros(len(ranks) * G * 128, dtype=torch.uint8).pin_memory()
    for s, r in enumerate(ranks):
        nat.lora_encode_tmap(tm_host[(s * G + 0) * 128:], arena.data_ptr() + bases[s] * 2, K, 3 * r, r * layer_units, L)
    tmaps = tm_host.cuda()
    # rows grouped by slot, with base-model rows in between
    seg = [(-1, 3), (0, 5), (2, T // 3), (1, 1), (3, T // 4)]
    rows = []
    for sl, n in seg:
        rows += [sl] * n
    rows = (rows + [1] * T)[:T]
    tl = ref.build_lora_tiles(rows, max_rows)
    tiles = torch.tensor(tl, device="cuda", dtype=torch.int32).view(-1, 4)
    pad = torch.full((7, 4), -1, device="cuda", dtype=torch.int32)
    tiles_padded = torch.cat([tiles, pad])
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    layer = 2
    offA = layer * layer_units
    offB = layer * layer_units + 3 * K
    nat.workspace().lora_v.zero_()      # columns past a slot's rank are never written; other tests leave values there
    vf = nat.lora_shrink_tiles(x, tiles_padded, tiles_padded.shape[0], max_rows, tmaps, G, 0, slot_rank, 3, layer, 64)
    torch.cuda.synchronize()
    nat.workspace().check_status()
    v = vf[:T].clone()
    v_ref = torch.zeros_like(v)
    ref.lora_shrink_tiles(x, tiles.cpu(), len(tl), max_rows, arena, slot_base, slot_rank, offA, 3, 64, v_ref)
    live = torch.tensor([s >= 0 for s in rows], device="cuda")
    assert _rel_err(v[live], v_ref[live]) < 4e-3
    y = torch.randn(T, N, device="cuda", dtype=torch.bfloat16)
    y_ref = y.clone()
    nat.lora_expand_tiles(vf[:T], tiles_padded, tiles_padded.shape[0], max_rows, arena, slot_base, slot_rank, offB, y, parts[0], parts[0] + parts[1])
    ref.lora_expand_tiles(v_ref, tiles.cpu(), len(tl), max_rows, arena, slot_base, slot_rank, offB, y_ref, parts[0], parts[0] + parts[1])
    nat.workspace().check_status()
    assert _rel_err(y, y_ref) < 5e-3
    # rows without a tile are untouched
    untouched = [i for i, s in enumerate(rows) if s < 0]
    assert torch.equal(y[untouched], y_ref[untouched])


@pytest.mark.parametrize("T,K,parts,ranks,layout", [(40, 1024, [512, 128, 128], [16, 48, 64, 32], "blocks"),
                                                    (256, 4096, [1024, 256, 256], [16, 16, 32, 64], "blocks"),
                                                    (700, 2048, [768, 768], [16, 32, 16, 64], "blocks"),
                                                    (300, 14336, [512], [16, 64, 32, 16], "blocks"),
                                                    # a prefill-sized step: every CTA walks several token tiles and rebuilds its unit list
                                                    (2304, 2048, [1536, 768], [16, 32, 16, 64], "runs"),
                                                    # another adapter on every row: more expand units per token tile than the list holds
                                                    (200, 1024, [512, 256], [16, 64, 32, 64], "alternating"),
                                                    # the same in a long step: one-row entries in the shrink units of four row groups
                                                    (600, 1024, [512, 256], [16, 64, 32, 64], "alternating")])
def test_gemm_with_lora_in_the_same_launch(nat, T, K, parts, ranks, layout):
    """Shrink items, base tiles and expand UMMAs in ONE launch of the GEMM kernel against fp32 PyTorch:
    x W^T + b + (x A_slot^T) B_slot^T per row, several adapters and ranks, base-model rows in between, rows of one adapter
    crossing 16-row and 256-row boundaries, rank 48 (a part that straddles two 128-row chunks of A_cat), two calls in a row."""
    torch.manual_seed(T + K)
    nparts, L = len(parts), 2
    N = sum(parts)
    layer_units = nparts * K + N
    bases, off = [], 0
    for r in ranks:
        bases.append(off)
        off += r * layer_units * L
        off = (off + 63) // 64 * 64
    arena = (torch.randn(off, device="cuda") * 0.05).to(torch.bfloat16)
    slot_base = torch.tensor(bases, device="cuda", dtype=torch.int64)
    slot_rank = torch.tensor(ranks, device="cuda", dtype=torch.int32)
    G = 5
    tm_host = torch.zeros(len(ranks) * 2 * G * 128, dtype=torch.uint8).pin_memory()
    for s, r in enumerate(ranks):
        nat.lora_encode_tmap(tm_host[(s * 2 * G + 0) * 128:], arena.data_ptr() + bases[s] * 2, K, nparts * r, r * layer_units, L)
        nat.lora_encode_tmap_b(tm_host[(s * 2 * G + G) * 128:], arena.data_ptr() + (bases[s] + r * nparts * K) * 2, r, N, r * layer_units, L)
    tmaps = tm_host.cuda()
    if layout == "blocks":
        seg = [(-1, 3), (0, 5), (2, T // 3), (1, 1), (3, T // 4), (-1, 2)]
        rows = []
        for sl, n in seg:
            rows += [sl] * n
        rows = (rows + [1] * T)[:T]
    elif layout == "runs":          # runs of 1 to 90 rows, adapters and base-model rows in turn
        g = torch.Generator().manual_seed(T)
        rows = []
        while len(rows) < T:
            rows += [int(torch.randint(-1, len(ranks), (1,), generator=g))] * int(torch.randint(1, 91, (1,), generator=g))
        rows = rows[:T]
    else:
        rows = [(i % (len(ranks) + 1)) - 1 for i in range(T)]
    tl = ref.build_lora_tiles(rows, 32)
    tiles = torch.cat([torch.tensor(tl, device="cuda", dtype=torch.int32).view(-1, 4), torch.full((9, 4), -1, device="cuda", dtype=torch.int32)])
    n0 = parts[0] if nparts > 1 else N
    n1 = parts[0] + parts[1] if nparts > 2 else N
    layer = 1
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    b = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    for call in range(2):
        x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
        lf = nat.LoraFused(tiles, tiles.shape[0], len(tl), tmaps, 2 * G, 0, G, slot_rank, slot_base, nparts, n0, n1, layer, max(ranks), arena, layer * layer_units, layer * layer_units + nparts * K)
        got = nat.gemm_lora_fused(x, w, lf, bias=b)
        assert got is not None
        torch.cuda.synchronize()
        nat.workspace().check_status()
        want = x.float() @ w.float().t() + b.float()
        bounds = [0, n0, n1, N] if nparts == 3 else ([0, n0, N] if nparts == 2 else [0, N])
        for t, sl in enumerate(rows):
            if sl < 0:
                continue
            r = ranks[sl]
            A = arena[bases[sl] + r * layer * layer_units:][: nparts * r * K].view(nparts * r, K).float()
            B = arena[bases[sl] + r * (layer * layer_units + nparts * K):][: N * r].view(N, r).float()
            v = (A @ x[t].float()).to(torch.bfloat16).float()            # the kernel rounds the shrink result to bf16
            for pp in range(nparts):
                lo, hi = bounds[pp], bounds[pp + 1]
                want[t, lo:hi] += B[lo:hi] @ v[pp * r:(pp + 1) * r]
        assert _rel_err(got, want) < 6e-3, call
        untouched = [i for i, s_ in enumerate(rows) if s_ < 0]
        base = nat.gemm(x, w, bias=b, mode=1)
        assert _rel_err(got[untouched], base[untouched]) < 1e-6


@pytest.mark.parametrize("T,K,parts,ranks,layout", [(2, 4096, [512, 128, 128], [16], "alternating"), (2, 14336, [512], [64], "alternating"),
                                                    (5, 3080, [768, 768], [16, 64, 32, 48], "alternating"), (6, 1000, [512], [32, 16], "alternating"),
                                                    (29, 4096, [4096, 1024, 1024], [16, 32], "runs"), (90, 2048, [512], [16], "runs"), (210, 4096, [2048, 512, 512], [16, 64, 32, 16], "blocks")])
def test_gemm_with_lora_of_few_units(nat, T, K, parts, ranks, layout):
    """Steps with fewer shrink units than CTAs, which share the K of each: one row, K of a part of a batch and of a ragged last one."""
    test_gemm_with_lora_in_the_same_launch(nat, T, K, parts, ranks, layout)


def _pair_tile(nat, T, N, K, rank=0):
    """Token tile of a product that pairs of CTAs take, 0 where single CTAs do."""
    ws, out = nat.workspace(), (ctypes.c_int * 4)()
    nat.load().lx_gemm_pair_plan(T, N, K, ws.num_sms, ws.num_sms // 2, ws.gemm_ws.numel(), rank, out)
    return out[0]


@pytest.mark.parametrize("T,K,parts,ranks,layout", [(200, 2048, [19264], [16, 32], "runs"), (257, 4096, [19072], [32, 16], "alternating"),
                                                    (300, 4096, [12800, 6208], [16], "alternating"), (520, 2048, [4096, 15168], [32, 16], "runs"),
                                                    (6000, 2048, [3264], [16, 32], "runs"), (5000, 2048, [4096, 1024, 320], [16, 32, 16, 32], "blocks")])
def test_gemm_with_lora_of_ragged_pairs(nat, T, K, parts, ranks, layout):
    """Pairs of CTAs whose last tile of 256 features is not full, the second CTA's half partly or all past the last feature: one part and several, a tile a
    pair and more."""
    assert _pair_tile(nat, T, sum(parts), K, max(ranks)) > 0 and sum(parts) % 256
    test_gemm_with_lora_in_the_same_launch(nat, T, K, parts, ranks, layout)


def test_leaving_out_the_expand_leaves_it_out_of_long_steps(nat, monkeypatch):
    """The measurement switch means the same where pairs of CTAs would take the product: the base product alone."""
    T, N, K, r, gen = 200, 19072, 2048, 16, torch.Generator("cuda").manual_seed(3)
    assert _pair_tile(nat, T, N, K, r) > 0
    x, w = (torch.randn(n, K, generator=gen, device="cuda").to(torch.bfloat16) / (1 if n == T else math.sqrt(K)) for n in (T, N))
    arena = torch.randn(r * (K + N), generator=gen, device="cuda").to(torch.bfloat16)
    maps = torch.zeros(2 * 128, dtype=torch.uint8).pin_memory()
    nat.lora_encode_tmap(maps, arena.data_ptr(), K, r, r * (K + N), 1)
    nat.lora_encode_tmap_b(maps[128:], arena.data_ptr() + r * K * 2, r, N, r * (K + N), 1)
    tiles = torch.tensor(ref.build_lora_tiles([0] * T, 32), device="cuda", dtype=torch.int32).view(-1, 4)
    rank, base = torch.tensor([r], device="cuda", dtype=torch.int32), torch.tensor([0], device="cuda", dtype=torch.int64)
    lf = nat.LoraFused(tiles, tiles.shape[0], tiles.shape[0], maps.cuda(), 2, 0, 1, rank, base, 1, N, N, 0, r, arena, 0, K)
    with_adapters, alone = nat.gemm_lora_fused(x, w, lf), nat.gemm(x, w, mode=1)
    monkeypatch.setenv("LORAX_LORA_SKIP", "2")
    assert _rel_err(nat.gemm_lora_fused(x, w, lf), alone) < 2 ** -8 and _rel_err(with_adapters, alone) > 1
    nat.workspace().check_status()


@pytest.mark.parametrize("form", ["fp8", "wq4"])
@pytest.mark.parametrize("T,K,parts,ranks", [(1, 512, [128], [16]), (5, 1024, [256, 128, 128], [16, 64]), (8, 512, [1024], [48]), (9, 2048, [512, 512], [32, 16]),
                                             (32, 4096, [384, 128, 128], [16, 32, 48, 64]), (77, 512, [256], [32, 16]), (256, 512, [16384], [16, 64]),
                                             (257, 512, [256, 256], [16])])
def test_quantised_products_add_the_adapters(nat, form, T, K, parts, ranks):
    """The delta of a short step, added in fp32 before the result is rounded, against the shrink's v in float64 on top of the product alone:
    rows of the base model in between, entries up to 32 rows, ranks of one to four 16s, with and without splits of K, and a step too long for it.
    Both sides round their sum to bf16, the reference the product before that: 2^-9 each."""
    from types import SimpleNamespace
    from lorax_b200.utils.quant_formats import quantize_weight
    N, nparts = sum(parts), len(parts)
    gen = torch.Generator("cuda").manual_seed(T + K)
    w = torch.randn(N, K, generator=gen, device="cuda").to(torch.bfloat16) / math.sqrt(K)
    x = torch.randn(T, K, generator=gen, device="cuda").to(torch.bfloat16)
    unit_off, bases, off = 64, [], 0
    for r in ranks:
        bases.append(off)
        off += r * (unit_off + N)
    arena = (torch.randn(off, generator=gen, device="cuda") * 0.5).to(torch.bfloat16)
    slots = [(i // 3) % (len(ranks) + 1) - 1 for i in range(T)] if T < 64 else [(i // 37) % (len(ranks) + 1) - 1 for i in range(T)]
    if T == 1:
        slots = [0]
    tl = ref.build_lora_tiles(slots, 32)
    table = torch.cat([torch.tensor(tl, device="cuda", dtype=torch.int32).view(-1, 4), torch.full((7, 4), -1, device="cuda", dtype=torch.int32)])
    tiles = SimpleNamespace(table=table, num_tiles=table.shape[0], max_rows=32, live=len(tl))
    v = nat.workspace().lora_v
    v[:T] = torch.randn(T, v.shape[1], generator=gen, device="cuda")
    n0 = parts[0] if nparts > 1 else N
    n1 = parts[0] + parts[1] if nparts > 2 else N
    i64 = torch.tensor(bases, device="cuda", dtype=torch.int64)
    epi = nat.LoraEpilogue(v, torch.tensor(slots, device="cuda", dtype=torch.int32), arena, i64, torch.tensor(ranks, device="cuda", dtype=torch.int32), unit_off, n0, n1)
    bias = torch.randn(N, generator=gen, device="cuda").to(torch.bfloat16)
    if form == "fp8":
        sw = torch.rand((N + 127) // 128, (K + 127) // 128, generator=gen, device="cuda") * 0.01 + 0.01
        q = (torch.randn(N, K, generator=gen, device="cuda") * 2).to(torch.float8_e4m3fn)
        run = lambda **kw: nat.gemm_fp8(x, q, sw, bias=bias, **kw)
    else:
        gq = quantize_weight(w, "hqq-4bit", 128)
        run = lambda **kw: nat.gemm_wq(x, gq, bias=bias, w_const=True, **kw)
    got, base = run(lora=(epi, tiles)), run()
    nat.workspace().check_status()
    want = base.double()
    edges = [0, n0, n1, N]
    for t, s in enumerate(slots):
        if s < 0:
            continue
        r = ranks[s]
        B = arena[bases[s] + r * unit_off:][: N * r].view(N, r).double()
        for part in range(nparts):
            lo, hi = edges[part], edges[part + 1] if part + 1 < nparts else N
            want[t, lo:hi] += B[lo:hi] @ v[t, part * r: (part + 1) * r].double()
    assert _rel_err(got, want) < 2 ** -8
    alone = [t for t, s in enumerate(slots) if s < 0]
    assert torch.equal(got[alone], base[alone])


@pytest.mark.parametrize("form,T,K,parts,ranks", [("fp8", 32, 512, [28672, 28672], [16, 64]), ("fp8", 32, 1024, [28672], [32, 48]), ("fp8", 144, 256, [4096], [16, 64, 32]),
                                                  ("wq4", 5, 512, [14336, 14336], [16, 64]), ("wq4", 32, 1024, [4096], [48, 16])])
def test_quantised_products_add_the_adapters_of_many_features(nat, form, T, K, parts, ranks):
    """At the ends of the range in which they do: several rows a warp of the kernel behind fp8 products among them."""
    test_quantised_products_add_the_adapters(nat, form, T, K, parts, ranks)


@pytest.mark.parametrize("T,K,parts,ranks", [(64, 512, [16384, 1024], [16, 64]), (96, 512, [256, 128], [16, 32, 64]), (255, 256, [4096], [48, 16]), (33, 1024, [260], [32])])
def test_quantised_products_add_the_adapters_of_prompts(nat, T, K, parts, ranks):
    """Entries of eight rows and more on average, whose rows are taken by fours: several such groups a warp and one, groups that end at an entry's end or the step's."""
    test_quantised_products_add_the_adapters(nat, "fp8", T, K, parts, ranks)


@pytest.mark.parametrize("T,N,K", [(193, 256, 64), (200, 6144, 4096), (256, 4096, 14336), (320, 28672, 256), (513, 256, 64), (545, 300, 200), (1000, 1000, 136), (2047, 640, 4096), (700, 4360, 72), (1024, 257, 64)])
def test_products_of_cta_pairs(nat, T, N, K):
    """Long steps at the edges of tiles, whole ones and shared: features that do not fill a tile of 256 or begin off 16 bytes in the output, ragged K, a last token tile of
    a few rows, with a bias.  fp32 sums, rounded to bf16: 2^-9."""
    g = torch.Generator("cuda").manual_seed(T + N)
    x = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") / math.sqrt(K)).to(torch.bfloat16)
    b = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    for bias in (b, None):
        got = nat.gemm(x, w, bias=bias)
        nat.workspace().check_status()
        want = x.double() @ w.double().t() + (0 if bias is None else bias.double())
        assert _rel_err(got, want) < 2 ** -8
    wide = torch.full((T, N + 24), 7.0, dtype=torch.bfloat16, device="cuda")      # rows of a wider buffer: nothing beside them is written
    nat.gemm(x, w, out=wide[:, :N])
    assert torch.equal(wide[:, :N], nat.gemm(x, w)) and (wide[:, N:] == 7).all()


@pytest.mark.parametrize("T,N,K", [(193, 28700, 4096), (256, 4100, 14336), (545, 6144, 8192), (700, 4360, 8200), (2047, 640, 14344), (3000, 2880, 2880), (4001, 4096, 1024)])
def test_products_that_pairs_of_ctas_take(nat, T, N, K):
    """The same where the plan prefers pairs: whole tiles in one wave and several, and all tiles shared."""
    assert _pair_tile(nat, T, N, K) > 0
    test_products_of_cta_pairs(nat, T, N, K)


@pytest.mark.parametrize("act", ["", "relu2", "swiglu"])
@pytest.mark.parametrize("lengths,n_w,K", [([0, 1, 31, 32, 33, 255, 256, 257, 511, 0], 256, 128), ([700, 3, 290], 512, 72), ([400], 768, 64)])
def test_expert_products_of_cta_pairs(nat, lengths, n_w, K, act):
    """Runs around the edges of tiles, empty ones among them, with every activation of the epilogue.  bf16 results: 2^-9."""
    g = torch.Generator("cuda").manual_seed(n_w + K)
    rows, E = sum(lengths), len(lengths)
    x = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(E, n_w, K, generator=g, device="cuda") / math.sqrt(K)).to(torch.bfloat16)
    seg = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), device="cuda", dtype=torch.int32)
    got = nat.moe_grouped_gemm(x, w, seg, 256, act=act)
    nat.workspace().check_status()
    at = 0
    for e, n in enumerate(lengths):
        y = x[at: at + n].double() @ w[e].double().t()
        if act == "relu2":
            y = y.clamp_min(0) ** 2
        elif act == "swiglu":
            y = torch.nn.functional.silu(y[:, ::2]) * y[:, 1::2]
        if n:
            assert _rel_err(got[at: at + n], y) < 2 ** -8, (e, n)
        at += n


@pytest.mark.parametrize("lengths,n_w", [([700, 3, 290, 0, 257], 256), ([33, 255, 512], 512)])
def test_gated_expert_products_of_cta_pairs(nat, lengths, n_w):
    """The gated epilogue of pairs, which take it from K of 3072 on."""
    assert nat.load().lx_moe_by_pairs(256, n_w, 3080, 2) == 1
    test_expert_products_of_cta_pairs(nat, lengths, n_w, 3080, "swiglu")


@pytest.mark.parametrize("num_sms", [2, 21, 148])
def test_expert_products_of_pairs_on_some_of_the_sms(nat, num_sms):
    """Fewer pairs walk more tiles each: the same bits."""
    g, E, n_w, K, rows = torch.Generator("cuda").manual_seed(num_sms), 3, 512, 256, 900
    x = torch.randn(rows, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(E, n_w, K, generator=g, device="cuda") / math.sqrt(K)).to(torch.bfloat16)
    seg, ws = torch.tensor([0, 400, 401, 900], device="cuda", dtype=torch.int32), nat.workspace()
    out = torch.empty(rows, n_w, dtype=torch.bfloat16, device="cuda")
    p = nat._ptr
    assert nat.load().lx_moe_grouped_gemm(p(x), K, p(w), K, p(out), n_w, p(seg), E, rows, rows, n_w, K, 300, 0, 0, 0, 0, p(ws.status), num_sms, nat._stream()) == 0
    ws.check_status()
    assert torch.equal(out, nat.moe_grouped_gemm(x, w, seg, 300))


@pytest.mark.parametrize("T,E,k,H,I,e0,e_local", [(7, 8, 2, 512, 256, 0, 8), (256, 8, 2, 1024, 768, 0, 8), (300, 8, 2, 512, 256, 2, 2),
                                                  (1500, 16, 4, 256, 128, 0, 16), (64, 4, 1, 256, 384, 1, 1)])
def test_moe_ffn_on_the_device(nat, T, E, k, H, I, e0, e_local):
    """Routing kernel, gather, grouped tcgen05 GEMMs and combine against the dense fp32 mixture of experts: softmax over all
    experts, top-k, renormalised weights; under expert parallelism (e_local < E) only the local experts' share."""
    torch.manual_seed(T + E)
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    wr = (torch.randn(E, H, device="cuda") * 0.3).to(torch.bfloat16)
    w13 = (torch.randn(e_local, 2 * I, H, device="cuda") / math.sqrt(H)).to(torch.bfloat16)
    w2 = (torch.randn(e_local, H, I, device="cuda") / math.sqrt(I)).to(torch.bfloat16)
    r = nat.moe_route(x, wr, k, e0, e_local)
    torch.cuda.synchronize()
    logits = x.float() @ wr.float().t()
    probs = torch.softmax(logits, -1)
    topv, topi = probs.topk(k, -1)
    # the kernel's choice may differ from torch's on near ties: compare the kept probability mass, and ids where the gap is clear
    gap = (probs.sort(-1, descending=True).values[:, k - 1] - probs.sort(-1, descending=True).values[:, k]) if k < E else torch.ones(T, device="cuda")
    clear = gap > 1e-3
    assert torch.equal(r.topk_ids[clear].long().sort(-1).values, topi[clear].sort(-1).values)
    wsum = r.topk_w.sum(-1)
    assert torch.allclose(wsum, torch.ones_like(wsum), atol=1e-5)
    seg = r.seg.tolist()
    assert seg[0] == 0 and all(a <= b for a, b in zip(seg, seg[1:]))
    ids = r.topk_ids.long()
    for e in range(e_local):
        assert seg[e + 1] - seg[e] == int((ids == e0 + e).sum())
    pos = r.pos.long()
    local = (ids >= e0) & (ids < e0 + e_local)
    assert (pos[~local] == -1).all() and (pos[local] >= 0).all()
    tok = torch.arange(T, device="cuda")[:, None].expand(T, k)
    assert torch.equal(r.xg[pos[local]], x[tok[local]])
    out = nat.moe_ffn(x, wr, w13, w2, k, e0, "silu")
    torch.cuda.synchronize()
    nat.workspace().check_status()
    # oracle with the kernel's own routing decision (so that near ties do not matter), dense fp32 experts
    want = torch.zeros(T, H, device="cuda")
    for e in range(e_local):
        sel = (ids == e0 + e)
        wt = (r.topk_w * sel).sum(-1)
        rows = wt > 0
        if rows.any():
            gu = x[rows].float() @ w13[e].float().t()
            a = (torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]).to(torch.bfloat16).float()
            y = (a @ w2[e].float().t()).to(torch.bfloat16).float()
            want[rows] += y * wt[rows, None]
    assert _rel_err(out, want) < 1.2e-2


@pytest.mark.parametrize("T,N,K", [(1, 256, 256), (16, 4096, 4096), (48, 1024, 14336), (100, 6144, 4096), (128, 384, 512),
                                   (300, 4096, 4096), (1000, 1024, 1024)])
def test_gemm_fp8_block128(nat, T, N, K):
    """Block-scaled e4m3 GEMM (128x128 weight scales, 1x128 activation scales) on tcgen05 kind::f8f6f4 against the
    PyTorch oracle that rounds both operands the same way and multiplies in fp32."""
    torch.manual_seed(T + N + K)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    x[:, ::97] *= 8.0                                  # a few outlier columns: the per-block scales must absorb them
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    b = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    wq, ws = ref.quantize_weight_fp8_block128(w)
    # the activation quantiser alone
    xq, sa = nat.quant_act_fp8(x)
    xq_ref, sa_ref = ref.quant_act_fp8(x)
    torch.cuda.synchronize()
    assert torch.allclose(sa[:, :T], sa_ref, rtol=1e-6, atol=0)
    a, b_ = xq.view(torch.float8_e4m3fn).float(), xq_ref.float()
    assert ((a - b_).abs() <= b_.abs() * 0.13 + 2e-3).all()          # x * (1 / s) against x / s: at most one e4m3 step apart
    assert (a != b_).float().mean().item() < 0.03
    saved = nat.FP8_EXPAND_MIN_TOKENS
    nat.FP8_EXPAND_MIN_TOKENS = 1 << 30            # the fp8 tensor-core kernel at every size
    try:
        out = nat.gemm_fp8(x, wq, ws, bias=b)
    finally:
        nat.FP8_EXPAND_MIN_TOKENS = saved
    torch.cuda.synchronize()
    nat.workspace().check_status()
    want = ref.gemm_fp8(x, wq, ws, bias=b)
    assert _rel_err(out, want) < 6e-3
    # long prefills expand the weights to bf16 and keep the activations in bf16: the oracle is x @ dequant(w)^T
    nat.FP8_EXPAND_MIN_TOKENS = 1
    try:
        out2 = nat.gemm_fp8(x, wq, ws, bias=b)
    finally:
        nat.FP8_EXPAND_MIN_TOKENS = saved
    torch.cuda.synchronize()
    nat.workspace().check_status()
    want2 = x.float() @ ref.dequantize_weight_fp8_block128(wq, ws).float().t()[:K, :N] + b.float() if False else \
        x.float() @ ref.dequantize_weight_fp8_block128(wq, ws)[:N, :K].float().t() + b.float()
    assert _rel_err(out2, want2) < 6e-3
    # and the quantised product is close to the bf16 one
    full = x.float() @ w.float().t() + b.float()
    assert _rel_err(out, full) < 6e-2


def test_fp8_weights_expanded_for_long_steps_carry_lora_in_the_gemm_launch(nat):
    """A long step over block-scaled e4m3 weights: the weights are expanded to bf16 once and the GEMM that carries the adapters runs
    over them; against fp32 PyTorch on the dequantised weights."""
    torch.manual_seed(11)
    T, K, parts, ranks = 640, 1024, [512, 256], [16, 32]
    nparts, N = len(parts), sum(parts)
    layer_units = nparts * K + N
    bases, off = [], 0
    for r in ranks:
        bases.append(off)
        off += (r * layer_units + 63) // 64 * 64
    arena = (torch.randn(off, device="cuda") * 0.05).to(torch.bfloat16)
    slot_base = torch.tensor(bases, device="cuda", dtype=torch.int64)
    slot_rank = torch.tensor(ranks, device="cuda", dtype=torch.int32)
    G = 5
    tm_host = torch.zeros(len(ranks) * 2 * G * 128, dtype=torch.uint8).pin_memory()
    for s_, r in enumerate(ranks):
        nat.lora_encode_tmap(tm_host[(s_ * 2 * G) * 128:], arena.data_ptr() + bases[s_] * 2, K, nparts * r, r * layer_units, 1)
        nat.lora_encode_tmap_b(tm_host[(s_ * 2 * G + G) * 128:], arena.data_ptr() + (bases[s_] + r * nparts * K) * 2, r, N, r * layer_units, 1)
    tmaps = tm_host.cuda()
    rows = [0] * 200 + [-1] * 40 + [1] * 400
    tl = ref.build_lora_tiles(rows, 32)
    tiles = torch.cat([torch.tensor(tl, device="cuda", dtype=torch.int32).view(-1, 4), torch.full((7, 4), -1, device="cuda", dtype=torch.int32)])
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / math.sqrt(K)
    wq, wscale = ref.quantize_weight_fp8_block128(w)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w16 = nat.fp8_expand(wq.view(torch.uint8), wscale)
    assert w16 is not None
    wd = ref.dequantize_weight_fp8_block128(wq, wscale)[:N, :K].float()
    assert _rel_err(w16.float(), wd) < 1e-2
    lf = nat.LoraFused(tiles, tiles.shape[0], len(tl), tmaps, 2 * G, 0, G, slot_rank, slot_base, nparts, parts[0], N, 0, max(ranks), arena, 0, nparts * K)
    got = nat.gemm_lora_fused(x, w16, lf)
    assert got is not None
    torch.cuda.synchronize()
    nat.workspace().check_status()
    want = x.float() @ wd.t()
    bounds = [0, parts[0], N]
    for sl in (0, 1):
        r = ranks[sl]
        idx = torch.tensor([t for t, s_ in enumerate(rows) if s_ == sl], device="cuda")
        A = arena[bases[sl]:][: nparts * r * K].view(nparts * r, K).float()
        B = arena[bases[sl] + r * nparts * K:][: N * r].view(N, r).float()
        v = (x[idx].float() @ A.t()).to(torch.bfloat16).float()
        for pp in range(nparts):
            lo, hi = bounds[pp], bounds[pp + 1]
            want[idx, lo:hi] += v[:, pp * r:(pp + 1) * r] @ B[lo:hi].t()
    assert _rel_err(got, want) < 6e-3
