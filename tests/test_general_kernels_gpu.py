"""Linears (fp32, bf16, int8), attention (general, prefill), activation rows, rotary embedding and the end of a step: kernels one by one,
at the edges of their tiles, splits, load widths and dispatch rules."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("M,N,K", [(1, 4, 4), (2, 7, 513), (3, 130, 2049), (4, 33, 512), (5, 4, 1030), (8, 200, 511), (9, 128, 256), (63, 129, 2048),
                                   (64, 127, 260), (65, 256, 1027), (129, 5, 4096), (400, 300, 777)])
def test_f32_linear_at_tile_and_split_edges(M, N, K, aligned):
    """Rows of the streaming kernel (up to 2, 4, 8), 64 x 128 tiles, K split over a cluster; 16-byte and 4-byte loads.  A sum of K
    products of random signs carries at most about sqrt(K) / 2 roundings of 6e-8 relative to its own size: 2e-6 at K = 4,096."""
    from mojo_linuxperiments_b200.ops import dense as D
    g = torch.Generator(device=DEV).manual_seed(M * 7919 + N)
    pad = 0 if aligned else 1
    ld = (K + 3) // 4 * 4 + pad
    x = torch.full((M, ld + pad), float("nan"), device=DEV)[:, pad:]           # what lies beyond K must not matter
    x[:, :K] = torch.randn((M, K), generator=g, device=DEV)
    w = torch.full((N, ld + pad), float("nan"), device=DEV)[:, pad:]
    w[:, :K] = torch.randn((N, K), generator=g, device=DEV) * K ** -0.5
    y = D.linear(x, D.DenseW(w, N, K))[:, :N]
    want = x[:, :K].double() @ w[:, :K].double().t()
    assert (y.double() - want).norm() <= 2e-6 * want.norm()
    assert (y.double() - want).abs().max() <= 2e-5 * want.abs().max().clamp_min(1.0)


def _us(fn, n=10):
    """Device time of a call in a captured run of ``n``, best of five."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(n):
            fn()
    t = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) * 1e3 / n)
    return min(t)


@pytest.mark.parametrize("M,N,K", [(9, 64, 33), (16, 100, 300), (33, 256, 96), (64, 130, 160), (65, 256, 256), (130, 1030, 224), (380, 512, 192)])
def test_f32_linear_with_fewer_than_eight_blocks_of_k_per_split(M, N, K):
    """Splits of one and two blocks, a last one that is partly filled; the bound of the longer sums."""
    from mojo_linuxperiments_b200.ops import dense as D
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x = D.rows(M, K, torch.float32, DEV)
    x.normal_(generator=g)
    W = torch.randn((N, K), generator=g, device=DEV) * K ** -0.5
    y = D.linear(x, D.DenseW.of(W, torch.float32, DEV))[:, :N]
    want = x[:, :K].double() @ W.double().t()
    assert (y.double() - want).norm() <= 2e-6 * want.norm()


@pytest.mark.parametrize("M,heads,n,k", [(1, 16, 512, 128), (2, 16, 512, 132), (3, 16, 516, 256), (4, 17, 500, 260), (8, 16, 512, 128), (8, 16, 511, 256), (8, 4, 2048, 64)])
def test_f32_heads_around_the_line_between_streaming_and_tiles(M, heads, n, k):
    from mojo_linuxperiments_b200.ops import dense as D
    g = torch.Generator(device=DEV).manual_seed(n + k)
    W = torch.randn((heads, n, k), generator=g, device=DEV) * k ** -0.5
    xk, yn = (k + 7) // 8 * 8, (n + 7) // 8 * 8
    x = torch.randn((M, heads * xk), generator=g, device=DEV)
    y = D.linear_heads(x, D.GroupedW.of(W, heads, torch.float32, DEV), xk, yn)
    want = torch.einsum("mhk,hnk->mhn", x.view(M, heads, xk)[..., :k].double(), W.double())
    assert (y.view(M, heads, yn)[..., :n].double() - want).norm() <= 2e-6 * want.norm()


def test_f32_linear_of_a_short_sum_takes_a_short_time():
    """K = 256 instead of 2,048 for few tiles: 6.3 us and 21 (20 and 21 where K was only split into eight blocks and more).  Eight rows over 16
    heads of 512 x 128: 1.0 times the time of nine rows (1.4 with a CTA for every four columns).  The bounds lie between."""
    from mojo_linuxperiments_b200.ops import dense as D
    x = torch.randn((65, 2048), device=DEV)
    short, long = D.DenseW.of(torch.randn((256, 256), device=DEV), torch.float32, DEV), D.DenseW.of(torch.randn((256, 2048), device=DEV), torch.float32, DEV)
    assert _us(lambda: D.linear(x, short)) < 0.6 * _us(lambda: D.linear(x, long))
    W, xh = D.GroupedW(torch.randn((16 * 512, 128), device=DEV), 16, 512, 128), torch.randn((9, 2048), device=DEV)
    assert _us(lambda: D.linear_heads(xh[:8], W, 128, 512)) < 1.2 * _us(lambda: D.linear_heads(xh, W, 128, 512))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("repeat", [1, 4])
@pytest.mark.parametrize("dk,dv,chunk", [(10, 6, None), (8, 8, 40), (130, 516, None), (36, 644, 100)])
def test_general_attention_with_uneven_head_sizes(dk, dv, chunk, repeat, dtype):
    """Head sizes that are no multiple of four, several parts of value dimensions, one to several blocks of keys per warp; few CTAs
    (eight warps) and many."""
    from mojo_linuxperiments_b200.ops import attention as A
    H, G, n, ps = 4, 2, 300, 16
    g = torch.Generator(device=DEV).manual_seed(dk)
    cache = A.PagedKVCache(32, G, ps, DEV, dk=dk, dv=dv, dtype=dtype)
    cache.data.normal_(generator=g)
    table = torch.randperm(32, generator=torch.Generator().manual_seed(1))[:20].to(torch.int32).view(1, 20).to(DEV)
    where = [0, 1, 31, 32, 33, 127, 128, 129, 255, n - 1] * repeat
    pos = torch.tensor(where, dtype=torch.int32, device=DEV)
    q = torch.randn((len(where), H * dk), generator=g, device=DEV).to(dtype)
    sink = torch.randn(H, generator=g, device=DEV)
    out = torch.full((len(where), H * dv), float("nan"), dtype=dtype, device=DEV)
    A.attn_paged(q, H, pos, torch.zeros_like(pos), cache, table, A.attn_spec(dk ** -0.5, chunk=chunk, sink=sink), out)
    page, row = table[0].long()[torch.arange(n, device=DEV) // ps], torch.arange(n, device=DEV) % ps
    k, v = cache.keys()[page, :, row].double(), cache.values()[page, :, row].double()
    for i, p in enumerate(where):
        lo = p // chunk * chunk if chunk else 0
        kk, vv = (t[lo:p + 1].repeat_interleave(H // G, 1) for t in (k, v))
        s = torch.einsum("hd,jhd->hj", q[i].double().view(H, dk), kk) * dk ** -0.5
        s = torch.cat([s, sink.double()[:, None]], 1).softmax(-1)[:, :-1]
        want = torch.einsum("hj,jhd->hd", s, vv).reshape(-1)
        # fp32 sums of up to 300 terms of size one; a bf16 result is rounded once (2^-9 of values up to 5)
        assert (out[i].double() - want).abs().max().item() < (1e-5 if dtype == torch.float32 else 1.2e-2), p


def _ok():
    from mojo_linuxperiments_b200.ops.workspace import default_workspace
    default_workspace(torch.device(DEV)).check_status()


@pytest.mark.parametrize("lens,hq,hkv", [([127, 128, 129], 8, 2), ([255, 256, 257, 1], 6, 2), ([130, 300], 3, 3), ([513, 64], 5, 1), ([200] * 40, 16, 4),
                                         ([1, 2, 700], 4, 4)])
def test_prefill_attention_pairs_heads_or_query_tiles(lens, hq, hkv):
    """Two heads of a KV head share a CTA; an odd number of them: two query tiles.  Tile edges, more items than CTAs, short
    sequences among long ones.  bf16 weights and outputs: 2^-8 of values up to 4."""
    from mojo_linuxperiments_b200.ops import attention as A
    g = torch.Generator(device=DEV).manual_seed(sum(lens))
    x = torch.randn((sum(lens), hq + 2 * hkv, 128), generator=g, device=DEV).to(torch.bfloat16)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    out = A.attn_prefill(x[:, :hq].contiguous(), x[:, hq:hq + hkv], x[:, hq + hkv:], cu, max(lens), kv_chunk=0)
    _ok()
    for part, o in zip(x.split(lens), out.split(lens)):
        q, k, v = (t.double() for t in (part[:, :hq], part[:, hq:hq + hkv].repeat_interleave(hq // hkv, 1), part[:, hq + hkv:].repeat_interleave(hq // hkv, 1)))
        s = torch.einsum("ihd,jhd->hij", q, k) * 128 ** -0.5
        s = s.masked_fill(torch.ones(s.shape[1:], dtype=torch.bool, device=DEV).triu(1), float("-inf")).softmax(-1)
        assert (o.double() - torch.einsum("hij,jhd->ihd", s, v)).abs().max().item() < 1.6e-2


@pytest.mark.parametrize("lens,hq,hkv", [([1], 2, 1), ([128], 4, 2), ([129, 256], 8, 2), ([1024], 32, 8), ([1025], 32, 8), ([128, 640, 641, 5], 8, 8), ([2049], 16, 4),
                                         ([300, 1, 129, 900] * 20, 3, 3)])
def test_prefill_attention_pairs_far_query_tiles(lens, hq, hkv):
    """A head's last query tile and its first share a CTA where all pairs fit one wave: one tile, a middle tile alone, sequences
    shorter than the longest, the sizes on both sides of a wave.  The weights of a row sum to 1, each is rounded
    to bf16 by at most 2^-9 of itself and the output by 2^-9 of values up to 4: 2^-8 * 4.  An empty sequence changes nothing."""
    test_prefill_attention_pairs_heads_or_query_tiles(lens, hq, hkv)
    from mojo_linuxperiments_b200.ops import attention as A
    x = torch.randn((sum(lens), hq + 2 * hkv, 128), device=DEV).to(torch.bfloat16)
    cu = [torch.tensor([0] + ls).cumsum(0).to(torch.int32).to(DEV) for ls in (lens, [0] + lens[:1] + [0] + lens[1:])]
    a, b = (A.attn_prefill(x[:, :hq].contiguous(), x[:, hq:hq + hkv], x[:, hq + hkv:], c, max(lens), kv_chunk=0) for c in cu)
    _ok()
    assert torch.equal(a, b)


@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("K", [128, 384, 512, 640, 2048, 4096, 8192, 8320, 14336, 16384])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_activation_rows_of_the_one_cta_form(mode, K, shift):
    """Chunks of four blocks, a last one that is partly filled, one and two chunks per warp; 16-byte and 8-byte accesses.  The whole
    numbers are those of the definition except where fp32 rounding moves a value across an edge (at most one step)."""
    from mojo_linuxperiments_b200.oracle import quant as Q
    from mojo_linuxperiments_b200.ops import linear as L
    M = 70
    g = torch.Generator(device=DEV).manual_seed(K + mode)
    W = K * (2 if mode == 3 else 1)
    x = torch.randn((M, W + 8), generator=g, device=DEV).to(torch.bfloat16)[:, shift:shift + W]
    x[3] = 0
    gamma = (1 + 0.1 * torch.randn(K, generator=g, device=DEV)).to(torch.bfloat16)
    res = torch.randn((M, K), generator=g, device=DEV).to(torch.bfloat16) if mode == 2 else None
    if res is not None:
        res[3] = 0
    base = None
    f = x.float()
    if mode == 3:
        f = Q.swiglu(x)
    elif mode == 2:
        base = (f + res.float()).to(torch.bfloat16)
        f = Q.rmsnorm(base, gamma, 1e-5)
    elif mode == 1:
        f = Q.rmsnorm(x, gamma, 1e-5)
    q, s = L.act_quant(x, mode=mode, gamma=gamma if mode in (1, 2) else None, residual=res)
    if base is not None:
        assert torch.equal(res, base)
    wq, ws = Q.rotate_quantize(f)
    assert (s - ws).abs().max() <= 3e-6 * ws.abs().max() and s[3] == 1.0
    d = (q.int() - wq.int()).abs()
    assert d.max() <= 1 and (d > 0).float().mean() < 2e-3


@pytest.mark.parametrize("tokens", [1, 1100])
@pytest.mark.parametrize("norm", [False, True])
def test_rotary_writes_the_same_with_narrow_accesses(tokens, norm):
    from mojo_linuxperiments_b200.ops import attention as A
    hq, hkv = 6, 2
    g = torch.Generator(device=DEV).manual_seed(tokens)
    W = (hq + 2 * hkv) * 128
    raw = torch.randn((tokens, W + 1), generator=g, device=DEV).to(torch.bfloat16)
    pos = (torch.arange(tokens, device=DEV) % 550).to(torch.int32)
    seq = (torch.arange(tokens, device=DEV) // 550).to(torch.int32)
    cos, sin = A.rope_tables(550, 1e4, DEV)
    w = (1 + 0.1 * torch.randn(128, generator=g, device=DEV)).to(torch.bfloat16) if norm else None
    got = []
    for x in (raw[:, 1:], raw[:, 1:].contiguous()):                  # odd pitch and start, then aligned rows
        cache = A.PagedKVCache(70, hkv, 16, DEV)
        k = torch.empty((tokens, hkv, 128), dtype=torch.bfloat16, device=DEV)
        q = A.rope_kv_write(x, pos, cos, sin, hq, hkv, k_out=k, cache=cache, page_table=torch.arange(70, dtype=torch.int32, device=DEV).view(2, 35),
                            seq_ids=seq, q_norm_w=w, k_norm_w=w)
        got.append((q, k, cache.data))
    _ok()
    for a, b in zip(*got):
        assert torch.equal(a, b)
    x = raw[:, 1:].double().view(tokens, -1, 128)[:, :hq + hkv]
    if norm:
        x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    c, s = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
    a, b = x[..., :64], x[..., 64:]
    want = torch.cat([a * c - b * s, b * c + a * s], -1)
    assert (torch.cat([got[0][0], got[0][1]], 1).double() - want).abs().max() < 2.5e-2      # one bf16 rounding of values up to 6


@pytest.mark.parametrize("bn", [-1, 256, 224, 192, 160, 128])
@pytest.mark.parametrize("M,N,K", [(129, 8, 16), (256, 264, 128), (257, 512, 272), (300, 1000, 1040), (1000, 2048, 896), (5000, 1288, 256)])
def test_int8_linear_of_two_ctas_per_tile(M, N, K, bn):
    """Edges of the 256-row tiles, channels that end inside a tile, K that ends inside a block, more tiles than pairs.  Whole
    sums, scaled in fp32 (two roundings of 2^-24) and rounded once to bf16, whose eight bits of significand leave 2^-8: 2^-7.99."""
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    sx, sw = torch.rand(M, generator=g, device=DEV) + 0.1, torch.rand(N, generator=g, device=DEV) + 0.1
    y = L.w8a8_gemm(x, sx, w, sw, force_mode=bn)
    _ok()
    want = (x.double() @ w.double().t()) * sx.double()[:, None] * sw.double()
    assert ((y.double() - want).abs() <= 2 ** -7.99 * want.abs()).all()


@pytest.mark.parametrize("force", [3, 64, 100, 127, 129, 200, 512])
@pytest.mark.parametrize("M", [100, 300])
def test_int8_linear_takes_a_number_that_names_no_tile_width_as_none(M, force):
    """Same kernel as without it above 128 tokens, the one-CTA kernel as with 0 below: the same bits either way."""
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M)
    x = torch.randint(-127, 128, (M, 512), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (520, 512), generator=g, device=DEV, dtype=torch.int8)
    sx, sw = torch.rand(M, generator=g, device=DEV), torch.rand(520, generator=g, device=DEV)
    want = L.w8a8_gemm(x, sx, w, sw, force_mode=-1 if M > 128 else 0)
    got = L.w8a8_gemm(x, sx, w, sw, force_mode=force)
    _ok()
    assert torch.equal(got, want)


@pytest.mark.parametrize("splits", [0, 1, 2, 3, 5, 8])
@pytest.mark.parametrize("M,N,K", [(65, 129, 1024), (96, 1000, 1040), (97, 384, 1792), (100, 4096, 1152), (128, 640, 2048), (128, 28672, 1024)])
def test_int8_linear_of_65_to_128_tokens(M, N, K, splits):
    """The 128-token form of the cluster kernel: ragged rows and channels, K that ends inside a block, every way to split.  Whole sums,
    scaled in fp32 (two roundings of 2^-24); bf16 rounds once more: 2^-7.99 of the value as above, 2^-22 for an fp32 result."""
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    sx, sw = torch.rand(M, generator=g, device=DEV) + 0.1, torch.rand(N, generator=g, device=DEV) + 0.1
    y = L.w8a8_gemm(x, sx, w, sw, force_mode=2, force_splits=splits)
    yf = L.w8a8_gemm(x, sx, w, sw, force_mode=2, force_splits=splits, out_dtype=torch.float32)
    _ok()
    want = (x.double() @ w.double().t()) * sx.double()[:, None] * sw.double()
    assert ((y.double() - want).abs() <= 2 ** -7.99 * want.abs()).all() and ((yf.double() - want).abs() <= 2 ** -22 * want.abs()).all()
    if splits == 0:
        assert torch.equal(L.w8a8_gemm(x, sx, w, sw), y)


@pytest.mark.parametrize("M,N,K,cluster", [(65, 6144, 2048, 0), (100, 6144, 4096, 0), (128, 8192, 4096, 0), (100, 12288, 4096, 0), (65, 18944, 4096, 0),
                                           (65, 57344, 4096, 0), (100, 128256, 4096, 0), (128, 512, 1024, 0), (100, 4096, 4096, 1), (128, 4096, 14336, 1),
                                           (100, 1024, 4096, 1), (65, 8192, 8192, 1), (100, 28672, 4096, 1), (128, 32000, 4096, 1)])
def test_int8_linear_of_65_to_128_tokens_goes_where_it_is_faster(M, N, K, cluster):
    """Shapes that one of the two kernels takes at least 1.1 times as long for as the other (1.03 for one to two tiles per SM)."""
    from mojo_linuxperiments_b200.ops import _lib
    assert _lib.lib().b200_w8a8_gemm_decode_takes(M, N, K, 148) == cluster


@pytest.mark.parametrize("M,N,K,splits", [(65, 129, 1024, 0), (100, 1000, 1040, 1), (128, 640, 2048, 3), (96, 4096, 1152, 0), (100, 20480, 256, 0)])
def test_int8_linear_of_65_to_128_tokens_has_the_bits_of_the_persistent_kernel(M, N, K, splits):
    """fp32 results, bf16 results in vectors and element by element: whole sums, scaled in the same order."""
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    sx, sw = torch.rand(M, generator=g, device=DEV) + 0.1, torch.rand(N, generator=g, device=DEV) + 0.1
    odd = N | 1
    for dtype, ld in ((torch.float32, N), (torch.bfloat16, (N + 7) // 8 * 8), (torch.bfloat16, odd)):
        got = []
        for force in (2, 0):
            y = torch.zeros((M, ld), dtype=dtype, device=DEV)
            L.w8a8_gemm(x, sx, w, sw, out=y[:, :N], force_mode=force, force_splits=splits if force == 2 else 0)
            got.append(y)
        _ok()
        n = N // 32 * 32 if dtype == torch.bfloat16 and ld % 8 == 0 and N % 8 else N        # a last part of a vector row is written by elements
        assert torch.equal(got[0][:, :n], got[1][:, :n]), (dtype, ld)


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("M,N,ld", [(20, 256, 258), (100, 256, 258), (100, 257, 259), (200, 256, 258), (100, 256, 257)])
def test_int8_linear_writes_rows_that_start_anywhere(M, N, ld, residual):
    """Results and residual rows whose first element lies on two bytes only, even and odd pitches, in every kernel of the range: the
    values of an aligned call (the scales may be multiplied in another order: one bf16 step), and nothing beside the rows."""
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randint(-127, 128, (M, 2048), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, 2048), generator=g, device=DEV, dtype=torch.int8)
    sx, sw = torch.rand(M, generator=g, device=DEV) + 0.1, torch.rand(N, generator=g, device=DEV) + 0.1
    buf, rbuf = (torch.full((M * ld + 1,), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    y, r = (b[1:].view(M, ld)[:, :N] for b in (buf, rbuf))
    r.copy_(1e5 * torch.randn((M, N), generator=g, device=DEV))
    L.w8a8_gemm(x, sx, w, sw, out=y, residual=r if residual else None)
    _ok()
    want = (x.double() @ w.double().t()) * sx.double()[:, None] * sw.double()
    bound = 2 ** -7.99 * want.abs()                      # one rounding to bf16, before or after the residual joins
    if residual:
        want = want + r.double()
        bound = bound + 2 ** -7.99 * want.abs()
    assert ((y.double() - want).abs() <= bound).all()
    assert buf[0] == 7.0 and (buf[1:].view(M, ld)[:, N:] == 7.0).all()


def test_linears_with_a_short_k_are_not_slower_than_a_cta_per_tile():
    """More than 128 tokens, K too short for what a pair of CTAs costs at its start and end (1.16 to 1.33 times as long before the rule
    looked at K): the call goes to the one-CTA tiles, which the right side forces."""
    from mojo_linuxperiments_b200.ops import dense as D
    from mojo_linuxperiments_b200.ops import linear as L
    x, w, s = D.rows(257, 256, torch.bfloat16, DEV), D.DenseW.of(torch.randn((1024, 256), device=DEV), torch.bfloat16, DEV), D.rows(257, 1024, torch.float32, DEV)
    x.normal_()
    s.zero_()
    for fn in (lambda force: D.linear(x, w, force=force), lambda force: D.linear_residual(x, w, s, 1e-6, None, None, force=force)):
        assert _us(lambda: fn(0)) < 1.1 * _us(lambda: fn(1))
    xq, sx = torch.randint(-127, 128, (2500, 256), device=DEV, dtype=torch.int8), torch.rand(2500, device=DEV)
    wq, sw = torch.randint(-127, 128, (16384, 256), device=DEV, dtype=torch.int8), torch.rand(16384, device=DEV)
    assert _us(lambda: L.w8a8_gemm(xq, sx, wq, sw)) < 1.1 * _us(lambda: L.w8a8_gemm(xq, sx, wq, sw, force_mode=0))


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 300])
def test_end_of_a_decode_step(rows):
    """Whole numbers: exact."""
    from mojo_linuxperiments_b200.ops import attention as A
    g = torch.Generator(device=DEV).manual_seed(rows)

    def ints(n, dtype=torch.int32):
        return torch.randint(0, 9999, (n,), generator=g, device=DEV, dtype=dtype)

    nxt, tokens, pos, lens, step = ints(rows, torch.int64), ints(rows, torch.int64), ints(rows), ints(rows), ints(4)
    active = ints(rows) % 2
    want = (pos + active, lens + active, step + 1)
    A.decode_advance(nxt, tokens, pos, lens, active, step)
    torch.cuda.synchronize()
    assert torch.equal(tokens, nxt) and all(torch.equal(a, b) for a, b in zip((pos, lens, step), want))


@pytest.mark.parametrize("bn", [0, 256, 224, 192, 160, 128])
@pytest.mark.parametrize("M,N,K", [(129, 4, 8), (256, 264, 136), (257, 518, 130), (300, 1000, 1040), (1000, 2048, 896), (5000, 1288, 256)])
def test_bf16_linear_of_two_ctas_per_tile(M, N, K, bn):
    """Edges of the 256-row tiles, channels that end inside a tile or a piece, K that ends inside a block, more tiles than pairs, all
    three epilogues.  K products of bf16 are summed in fp32: K 2^-24 of the sum of their magnitudes at most; a bf16 result
    rounds once more (2^-9 of the value, 2-norm below 4e-3)."""
    from mojo_linuxperiments_b200.ops import dense as D
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = D.rows(M, K, torch.bfloat16, DEV)
    x[:, :K].normal_(generator=g)
    W = torch.randn((N, K), generator=g, device=DEV).to(torch.bfloat16)
    w, xd, wd = D.DenseW.of(W, torch.bfloat16, DEV), x[:, :K].double(), W.double()
    want, bound = xd @ wd.t(), K * 2 ** -24 * (xd.abs() @ wd.abs().t())
    y, y16 = D.linear(x, w, out_dtype=torch.float32, force=-bn)[:, :N], D.linear(x, w, force=-bn)[:, :N]
    s = D.rows(M, N, torch.float32, DEV)
    s.normal_(generator=g)
    base = s[:, :N].double()
    D.linear_residual(x, w, s, 1.0, None, None, force=-bn)
    glu = D.linear_glu(x, w, 7.0, force=-bn)[:, :N // 2].double()
    _ok()
    assert ((y.double() - want).abs() <= bound).all()
    assert ((s[:, :N].double() - base - want).abs() <= bound + 2 ** -23 * (base.abs() + want.abs())).all()
    a, u = want[:, 0::2].clamp(max=7.0), want[:, 1::2].clamp(-7.0, 7.0)
    for got, ref in ((y16.double(), want), (glu, a * torch.sigmoid(1.702 * a) * (u + 1))):
        assert (got - ref).norm() <= 4e-3 * ref.norm()


@pytest.mark.parametrize("splits", range(9))
@pytest.mark.parametrize("M,N,K", [(1, 4, 32), (9, 128, 33), (16, 129, 511), (127, 5, 512), (128, 300, 1027), (129, 256, 2049), (400, 130, 4096), (40, 66, 2048)])
def test_f32_linear_in_three_bf16_parts(M, N, K, splits):
    """Every split (0: as the rule has it), edges of the 128 x 128 tiles, of blocks of 32 k, of the periods of 256 and 1,024 k, one block per split;
    what lies beyond K or M does not matter.  Splitting is exact but for products of 2^-34, a sum of 32 k is cut off at 2^-23, sums of sums are
    rounded: no further from 64 bits than the sums of the CUDA cores for the calls that go there.  Forced: two cuts per block, each at most 2^-23
    and half of that on average, 1.2e-7 of the blocks' sums, which add up where all products have one sign; a dozen roundings of the sum so far,
    0.3e-7 each and half of it large on average, as a root of squares 0.6e-7: 1.5e-7 together for the lengths that the rule leaves out."""
    from mojo_linuxperiments_b200.ops import dense as D
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    for kind in ("signs", "positive", "sizes", "last bits"):
        X, W = torch.randn((M, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV) * K ** -0.5
        if kind == "positive":
            X, W = X.abs(), W.abs()
        if kind == "sizes":
            X = X * torch.exp2(torch.randint(-20, 20, (M, K), generator=g, device=DEV).float())
        if kind == "last bits":                            # the second and third parts are as large as they can be: x2 w3 + x3 w2 is 2^-24 of x w
            X, W = 1.0038833618164062 * X.sign(), 1.0038833618164062 * W.sign()
        x = torch.full((M + 1, (K + 3) // 4 * 4 + 4), float("nan"), device=DEV)[:M]
        x[:, :K] = X
        w = torch.full((N, (K + 3) // 4 * 4), float("nan"), device=DEV)
        w[:, :K] = W
        want = X.double() @ W.double().t()

        def off(force):
            y = D.linear(x, D.DenseW(w, N, K), force=force)[:, :N]
            return ((y.double() - want).norm() / want.norm()).item()

        most = 0.0 if splits == 0 else 1.5e-7 if K < 2048 else 1.2e-7 if kind == "positive" else 0.0
        assert off(splits) <= max(off(-1), most), kind


def test_f32_linear_of_nothing_but_nan_takes_no_longer_than_on_the_cuda_cores():
    """Outputs that are not finite are computed again; a row of NaN, as a broken input makes all of them, is not.  Measured 0.4 of the CUDA cores'
    time; with a serial sum per output 77 times as long."""
    from mojo_linuxperiments_b200.ops import dense as D
    x, w = torch.full((256, 2048), float("nan"), device=DEV), D.DenseW.of(torch.randn((1024, 2048), device=DEV), torch.float32, DEV)
    ms = {}
    for force in (2, -1):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(200000)
            a.record()
            y = D.linear(x, w, force=force)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        assert torch.isnan(y).all()
        ms[force] = sorted(times)[2]
    assert ms[2] < 2 * ms[-1], ms


@pytest.mark.parametrize("M,N,K", [(9, 256, 2048), (70, 2050, 2048), (300, 520, 2500)])
def test_f32_linears_with_their_epilogues_on_the_tensor_cores(M, N, K):
    """The calls that the rule sends there, with a gate and up (interleaved columns) and with a residual, against 64 bits and the CUDA cores: 2e-7 of
    the sum, tanh and the exponential two units more."""
    from mojo_linuxperiments_b200.ops import _lib
    from mojo_linuxperiments_b200.ops import dense as D
    assert _lib.lib().b200_f32_gemm_tc_takes(M, N, K) == 1
    g = torch.Generator(device=DEV).manual_seed(M)
    x = D.rows(M, K, torch.float32, DEV)
    x.normal_(generator=g)
    W = torch.randn((N, K), generator=g, device=DEV) * K ** -0.5
    w = D.DenseW.of(W, torch.float32, DEV)
    v = x[:, :K].double() @ W.double().t()
    gate, up = v[:, 0::2].clamp(max=1.0), v[:, 1::2].clamp(-1.0, 1.0)
    glu = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    s0 = torch.randn((M, D.padded(N)), generator=g, device=DEV)
    norm = D.DynamicTanh.of(0.7, torch.randn(N, generator=g, device=DEV), torch.randn(N, generator=g, device=DEV), DEV)
    new = s0[:, :N].double() + 0.5 * v
    for force in (0, -1):
        assert (D.linear_glu(x, w, 1.0, force=force)[:, :N // 2].double() - glu).norm() <= 5e-7 * glu.norm()
        s, out = s0.clone(), D.rows(M, N, torch.float32, DEV)
        D.linear_residual(x, w, s, 0.5, norm, out, force=force)
        want = torch.tanh(norm.alpha * new) * norm.w[:N].double() + norm.b[:N].double()
        assert (s[:, :N].double() - new).norm() <= 3e-7 * new.norm() and (out[:, :N].double() - want).norm() <= 5e-7 * want.norm()
    _ok()


def test_f32_linear_in_three_parts_where_it_is_not_finite():
    from mojo_linuxperiments_b200.ops import dense as D
    g = torch.Generator(device=DEV).manual_seed(5)
    x = D.rows(130, 640, torch.float32, DEV)
    x.normal_(generator=g)
    W = torch.randn((200, 640), generator=g, device=DEV)
    inf = float("inf")
    x[7] *= 1e30
    x[:, 630], W[:, 0] = 1e-3, W[:, 0] * 1e-3
    x[3, 7], x[5, 9], x[7, 3], x[8, 1], W[9, 1] = inf, float("nan"), -inf, 0.0, inf
    x[11] = inf
    x[129, 0], W[77, 630] = 3.4e38, -3.4e38                   # round to infinity in bf16; every sum of them is finite
    a, b = (D.linear(x, D.DenseW.of(W, torch.float32, DEV), force=f)[:, :200] for f in (2, -1))
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b)) and torch.equal(a[torch.isinf(a)], b[torch.isinf(b)])
    fine = torch.isfinite(b)
    assert ((a - b).abs() <= 1e-5 * x.abs().nan_to_num(0, 0, 0).amax(1, keepdim=True).clamp_min(1.0) * W.abs().nan_to_num(0, 0, 0).amax(1))[fine].all()
    assert torch.isnan(a[8, 9]) and fine[129, 1] and fine[0, 77]


@pytest.mark.parametrize("H,G,dk,dv,chunk,spans", [(8, 2, 128, 128, None, [(0, 127), (0, 128), (0, 129), (37, 300)]), (6, 2, 64, 96, 200, [(0, 257), (150, 260), (5, 1)]),
                                                   (3, 3, 40, 16, 70, [(0, 513), (64, 130)]), (16, 4, 128, 128, 512, [(300 * (i % 2), 200 + 40 * i) for i in range(12)]),
                                                   (5, 1, 8, 128, 128, [(100, 400), (0, 256)]), (16, 4, 128, 128, None, [(0, 128), (300, 100)]),
                                                   (16, 4, 64, 64, 200, [(100 * i, 128 - 9 * i) for i in range(10)])])
def test_paged_prefill_attention_pairs_heads_or_query_tiles(H, G, dk, dv, chunk, spans):
    """(first position, tokens) of portions.  Two heads of a KV head share a CTA; an odd number of them: two query tiles, the second of which
    may start in a later chunk; one query tile each of a few portions: a head alone.  Tile edges, portions that continue, more items than CTAs.  bf16 weights and outputs: 2^-8 of values up to 4."""
    from mojo_linuxperiments_b200.ops import attention as A
    ps, B = 16, len(spans)
    g = torch.Generator(device=DEV).manual_seed(dk + B)
    per = max((a + n + ps - 1) // ps for a, n in spans)
    cache = A.PagedKVCache(B * per + 3, G, ps, DEV, dk=dk, dv=dv, dtype=torch.bfloat16)
    cache.data.normal_(generator=g)
    table = torch.randperm(B * per, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(B, per).to(DEV)
    lens = [n for _, n in spans]
    pos = torch.cat([torch.arange(a, a + n, dtype=torch.int32) for a, n in spans]).to(DEV)
    sid = torch.cat([torch.full((n,), b, dtype=torch.int32) for b, (_, n) in enumerate(spans)]).to(DEV)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    q = torch.randn((sum(lens), H * dk), generator=g, device=DEV).to(torch.bfloat16)
    sink, gate = torch.randn(H, generator=g, device=DEV), torch.randn((sum(lens), 8 * ((H + 7) // 8)), generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((sum(lens), H * dv), float("nan"), dtype=torch.bfloat16, device=DEV)
    A.attn_prefill_paged(q, H, pos, sid, cu, max(lens), cache, table, A.attn_spec(dk ** -0.5, chunk=chunk, sink=sink, gate=gate), out)
    _ok()
    for b, (a, n) in enumerate(spans):
        at, end = cu[b].item(), a + n
        j = torch.arange(end, device=DEV)
        k, v = (t[table[b].long()[j // ps], :, j % ps].double().repeat_interleave(H // G, 1) for t in (cache.keys(), cache.values()))
        i = torch.arange(a, end, device=DEV)
        seen = j[None] <= i[:, None]
        if chunk:
            seen &= j[None] // chunk == i[:, None] // chunk
        s = torch.einsum("ihd,jhd->hij", q[at:at + n].double().view(n, H, dk), k) * dk ** -0.5
        s = torch.cat([s.masked_fill(~seen, -float("inf")), sink.double()[:, None, None].expand(H, n, 1)], 2).softmax(-1)[..., :-1]
        want = torch.einsum("hij,jhd->ihd", s, v) * torch.sigmoid(gate[at:at + n, :H].double())[..., None]
        assert (out[at:at + n].double() - want.reshape(n, H * dv)).abs().max().item() < 1.6e-2, (b, a, n)


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M", [1, 15, 16, 17, 31, 33, 63, 64, 65, 99, 128])
def test_w8a8_decode_exchange(M, splits):
    """Partial sums of every split, odd and even numbers of tokens, slices that are no multiple of four channels, a last tile that is partly
    filled: whole numbers until the scales (two fp32 roundings) and the store (bf16, 2^-8)."""
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M * 8 + splits)
    N, K = 328, 1168
    x = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=DEV, generator=g)
    w = torch.randint(-127, 128, (N, K), dtype=torch.int8, device=DEV, generator=g)
    sx, sw = torch.rand(M, device=DEV, generator=g), torch.rand(N, device=DEV, generator=g)
    want = (x.double() @ w.double().t()) * sx.double()[:, None] * sw.double()
    y = L.w8a8_gemm(x, sx, w, sw, force_mode=2, force_splits=splits)
    _ok()
    assert ((y.double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -22)).all()


@pytest.mark.parametrize("M", [9, 16, 64, 380])
def test_f32_linears_that_hand_one_buffer_on(M):
    """Read, rewritten in place, read again, launch after launch, as the stream of a model's layers: captured and replayed, with kernels that
    start before their input is there, the bits of the same launches one at a time.  A row that L1 still holds from the launch
    before would show."""
    from mojo_linuxperiments_b200.ops import dense as D
    g, d, layers = torch.Generator(device=DEV).manual_seed(M), 2048, 4
    w = [[D.DenseW.of(torch.randn((d, d), generator=g, device=DEV) * d ** -0.5, torch.float32, DEV) for _ in range(2)] for _ in range(layers)]
    norm = D.DynamicTanh.of(0.5, torch.randn(d, generator=g, device=DEV), torch.randn(d, generator=g, device=DEV), DEV)
    x0 = torch.empty((M, d), device=DEV)
    x, h = torch.empty_like(x0), torch.empty_like(x0)

    def run(after=lambda: None):
        x.copy_(x0)
        h.copy_(x0)
        for a, b in w:
            y = D.linear(h, a)
            after()
            D.linear_residual(y, b, x, 0.7, norm, h)
            after()
        return D.linear(h, w[0][0])

    side = torch.cuda.Stream()
    x0.normal_(generator=g)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = run()
    for _ in range(20):
        x0.normal_(generator=g)
        graph.replay()
        got = x.clone(), h.clone(), y.clone()
        want_y = run(torch.cuda.synchronize)
        assert torch.equal(got[0], x) and torch.equal(got[1], h) and torch.equal(got[2], want_y)
    _ok()


@pytest.mark.parametrize("prologue", [False, True])
@pytest.mark.parametrize("M", [1, 5, 16, 17, 40, 64])
def test_token_scales_of_launch_after_launch(M, prologue):
    """Every split, launches that follow each other with other scales: a finished value takes those of its own launch."""
    from mojo_linuxperiments_b200.ops import linear as L
    from mojo_linuxperiments_b200.ops.workspace import default_workspace
    g = torch.Generator(device=DEV).manual_seed(M)
    N, K, n = 1152, 2048, 7
    w = torch.randint(-127, 128, (N, K), dtype=torch.int8, device=DEV, generator=g)
    sw = torch.rand(N, device=DEV, generator=g)
    x = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=DEV, generator=g)
    xb = torch.randn((M, K), device=DEV, generator=g).to(torch.bfloat16)
    scales = [torch.rand(M, device=DEV, generator=g) * 10.0 ** i for i in range(n)]
    rows_ = [xb * 4.0 ** i for i in range(n)]
    acc = x.double() @ w.double().t() * sw.double()

    def run():
        if prologue:                                     # the launch's own quantiser CTAs publish the scales; powers of four: the same int8 rows
            default_workspace(torch.device(DEV)).next_step()
            return [L.fused_linear(r, w, sw) for r in rows_]
        return [L.w8a8_gemm(x, s, w, sw, force_mode=2, force_splits=2 + i) for i, s in enumerate(scales)]

    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for _ in range(30):
        graph.replay()
        for i, y in enumerate(out):
            if prologue:
                assert torch.equal(y, out[0] * 4.0 ** i)
            else:
                want = acc * scales[i].double()[:, None]
                assert ((y.double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -22)).all()
    _ok()


@pytest.mark.parametrize("H,G", [(3, 3), (4, 2)])
def test_paged_prefill_attention_drops_the_query_tile_without_pages(H, G):
    """A table that ends inside the second query tile of a portion: that tile is reported and left out, the first one is computed, with pairs
    of heads and with pairs of query tiles."""
    from mojo_linuxperiments_b200.ops import attention as A
    g = torch.Generator(device=DEV).manual_seed(H)
    n, dk, ps, pages = 250, 64, 16, 10
    cache = A.PagedKVCache(16, G, ps, DEV, dk=dk, dv=dk, dtype=torch.bfloat16)
    cache.data.normal_(generator=g)
    table = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, pages)
    q = torch.randn((n, H * dk), generator=g, device=DEV).to(torch.bfloat16)
    pos, sid, out = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV), {}
    for rows in (128, n):
        cu = torch.tensor([0, rows], dtype=torch.int32, device=DEV)
        out[rows] = torch.full((n, H * dk), 7.0, dtype=torch.bfloat16, device=DEV)
        A.attn_prefill_paged(q, H, pos, sid, cu, rows, cache, table, A.attn_spec(dk ** -0.5), out[rows])
        if rows == n:
            with pytest.raises(RuntimeError, match="attn_prefill_paged"):
                _ok()
        else:
            _ok()
    assert torch.equal(out[n][:128], out[128][:128]) and (out[n][128:] == 7.0).all() and not (out[n][:128] == 7.0).all()


def test_f32_linear_takes_the_values_of_force_that_choose_a_bf16_tile():
    from mojo_linuxperiments_b200.ops import dense as D
    x, w = torch.randn((16, 2048), device=DEV), D.DenseW.of(torch.randn((200, 2048), device=DEV), torch.float32, DEV)
    want = D.linear(x, w)[:, :200]
    for force in (9, 64, 256, -64, -256):
        assert torch.equal(D.linear(x, w, force=force)[:, :200], want), force


@pytest.mark.parametrize("M", [33, 48, 49, 64])
@pytest.mark.parametrize("N,K", [(512, 4096), (1920, 1024), (4352, 1040), (12928, 1024), (18944, 2048), (19072, 512)])
def test_decode_linears_with_either_ring(M, N, K):
    """Grids on both sides of a CTA per multiprocessor, whole tiles and split ones.  int8: whole numbers until the scales (two fp32 roundings) and the
    store (bf16, 2^-8).  bf16: products are exact, fp32 sums of K terms of random signs are off by less than 1e-5 of the largest, the store 2^-8."""
    from mojo_linuxperiments_b200.ops import dense as D
    from mojo_linuxperiments_b200.ops import linear as L
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=DEV, generator=g)
    w = torch.randint(-127, 128, (N, K), dtype=torch.int8, device=DEV, generator=g)
    sx, sw = torch.rand(M, device=DEV, generator=g), torch.rand(N, device=DEV, generator=g)
    want = (x.double() @ w.double().t()) * sx.double()[:, None] * sw.double()
    y = L.w8a8_gemm(x, sx, w, sw)
    assert ((y.double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -22)).all()
    xb = torch.randn((M, K), device=DEV, generator=g).to(torch.bfloat16)
    wb = (torch.randn((N, K), device=DEV, generator=g) * K ** -0.5).to(torch.bfloat16)
    want = xb.double() @ wb.double().t()
    y = D.linear(xb, D.DenseW.of(wb, torch.bfloat16, DEV))[:, :N].double()
    assert ((y - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5 * want.abs().max()).all()
    _ok()
