"""Every CUDA kernel alone against its plain PyTorch statement (tests/plain_ops.py),
at sizes other than the tiny models': widths that are no power of two, head
sizes 16 to 256, group sizes 1 to 8, shuffled pages, a window, and inputs made
so that a wrong key, page or row shows."""
import math

import pytest
import torch

import plain_ops

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def ops():
    import llm_b200.ops as o
    return o


def tol(dtype, scale=1.0):
    return dict(atol=(2e-5 if dtype == torch.float32 else 2e-2) * scale,
                rtol=1e-5 if dtype == torch.float32 else 2e-2)


def randn(*shape, dtype=torch.float32, seed=0, scale=1.0):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=gen) * scale).to(dtype).to(DEV)


@pytest.mark.parametrize("dtype", DTYPES)
def test_embed(dtype):
    table = randn(301, 72, dtype=dtype)
    tokens = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32, device=DEV)
    assert torch.equal(ops().embed(tokens, table), plain_ops.embed(tokens, table))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden", [64, 96, 1000, 4096])
def test_rmsnorm(dtype, hidden):
    x = randn(7, hidden, seed=1, scale=3.0)
    x[3] *= 1e-3                         # a row where eps matters
    gain = 1.0 + randn(hidden, seed=2, scale=0.1)
    rows = torch.tensor([6, 0, 3, 3], dtype=torch.int32, device=DEV)
    for r in (None, rows):
        got = ops().rmsnorm(x, gain, 1e-5, dtype, r)
        want = plain_ops.rmsnorm(x, gain, 1e-5, dtype, r)
        assert torch.allclose(got.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_swiglu(dtype):
    gu = randn(5, 2 * 172, dtype=dtype, seed=3, scale=2.0)
    got = ops().swiglu(gu)
    assert torch.allclose(got.float(), plain_ops.swiglu(gu).float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("m,n,k", [(1, 96, 64), (7, 172, 64), (65, 100, 172), (129, 384, 96),
                                   (193, 130, 250), (33, 1000, 80)])
def test_linear(dtype, m, n, k):
    a = randn(m, k, dtype=dtype, seed=4)
    w = randn(n, k, dtype=dtype, seed=5, scale=0.1)
    bias = randn(n, seed=6)
    got = ops().linear(a, w, bias)
    want = plain_ops.linear(a, w, bias)
    assert torch.allclose(got.float(), want.float(), **tol(dtype, math.sqrt(k) / 8))
    # 32-bit output (the head) and accumulation into the residual stream
    got32 = ops().linear(a, w, out_dtype=torch.float32)
    assert torch.allclose(got32, plain_ops.linear(a, w, out_dtype=torch.float32), **tol(torch.float32, math.sqrt(k)))
    residual = randn(m, n, seed=7)
    expect = plain_ops.linear(a, w, bias, residual=residual.clone())
    ops().linear(a, w, bias, residual=residual)
    assert torch.allclose(residual, expect, **tol(torch.float32, math.sqrt(k)))


@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (8, 6144, 4096), (8, 1000, 200), (5, 72, 1032),
                                   (16, 4096, 14336), (17, 100, 1024), (33, 520, 2048),
                                   (64, 4100, 4096)])
@pytest.mark.parametrize("variant", ["gemm_skinny", "gemm_tc"])
def test_linear_decode_kernel(m, n, k, variant):
    """The split-K decode products (mma.sync and tcgen05): sizes with one and many
    splits, tails in N, K and M, called twice so that the tile counters must have
    been left at zero."""
    from llm_b200.ops import tactics
    if variant == "gemm_skinny":
        tactics.disable("gemm_tc")
    try:
        assert tactics.choose_linear(m, n, k, torch.bfloat16, torch.bfloat16, k) == variant
        _check_decode_product(m, n, k)
        assert ops().tensor_core_status() == 0
    finally:
        tactics.enable("gemm_tc")


def _check_decode_product(m, n, k):
    a = randn(m, k, dtype=torch.bfloat16, seed=80)
    w = randn(n, k, dtype=torch.bfloat16, seed=81, scale=0.05)
    bias = randn(n, seed=82)
    want = plain_ops.linear(a, w, bias, out_dtype=torch.float32)
    scale = float(want.abs().max())
    for _ in range(2):
        got = ops().linear(a, w, bias, out_dtype=torch.float32)
        assert float((got - want).abs().max()) <= 2e-3 * scale
    got16 = ops().linear(a, w, bias)
    assert float((got16.float() - want).abs().max()) <= 1e-2 * scale
    residual = randn(m, n, seed=83)
    expect = residual + want
    ops().linear(a, w, bias, residual=residual)
    assert float((residual - expect).abs().max()) <= 2e-3 * scale
    # the same rows alone and in the batch: the same split and order, bit-equal
    alone = ops().linear(a[:1].contiguous(), w, bias, out_dtype=torch.float32)
    assert torch.equal(alone[0], got[0])


@pytest.mark.parametrize("m,n,k", [(65, 256, 64), (128, 128, 128), (129, 300, 200), (200, 1000, 520),
                                   (513, 6144, 4096), (2048, 4096, 1024), (70, 72, 72),
                                   (300, 4104, 2048), (256, 4096, 4096), (1000, 2304, 1536),
                                   (140, 19200, 128), (2500, 8192, 192)])
def test_linear_tensor_core_kernel(m, n, k):
    """tcgen05 product for more than 64 tokens: tile edges in M, N and K, on each of its kernels: weights on the 128-row side with
    several token tiles and split K (256 x 4096), on the pairs' row side (513 x 6144, 300 x 4104), 256 x 256 tiles on pairs
    of SMs (2500 x 8192)."""
    from llm_b200.ops import tactics
    assert tactics.choose_linear(m, n, k, torch.bfloat16, torch.bfloat16, k) == "gemm_tc"
    a = randn(m, k, dtype=torch.bfloat16, seed=84)
    w = randn(n, k, dtype=torch.bfloat16, seed=85, scale=0.05)
    bias = randn(n, seed=86)
    want = plain_ops.linear(a, w, bias, out_dtype=torch.float32)
    scale = float(want.abs().max())
    got = ops().linear(a, w, bias, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert ops().tensor_core_status() == 0
    assert float((got - want).abs().max()) <= 2e-3 * scale
    got16 = ops().linear(a, w, bias)
    assert float((got16.float() - want).abs().max()) <= 1e-2 * scale
    residual = randn(m, n, seed=87)
    expect = residual + want
    ops().linear(a, w, bias, residual=residual)
    assert float((residual - expect).abs().max()) <= 2e-3 * scale
    # a strided view as input (the query part of a fused projection)
    wide = randn(m, k + 64, dtype=torch.bfloat16, seed=88)
    view = wide[:, :k]
    got = ops().linear(view, w, out_dtype=torch.float32)
    assert float((got - plain_ops.linear(view, w, out_dtype=torch.float32)).abs().max()) <= 2e-3 * scale


@pytest.mark.parametrize("m,f,k", [(1, 64, 64), (8, 14336, 4096), (5, 208, 72), (64, 320, 128),
                                   (70, 320, 128), (300, 1024, 520), (2048, 1024, 256),
                                   (8, 320, 1024), (40, 320, 1024), (512, 2048, 2048)])
def test_linear_with_gated_epilogue(m, f, k):
    """silu(gate) * up in the epilogue of the tensor-core product, both orientations,
    against the product followed by the plain activation. The last two shapes split K: the
    activation is then applied where the splits are summed (by the last block of a tile at 8
    tokens, by the sum kernel at 40)."""
    a = randn(m, k, dtype=torch.bfloat16, seed=96)
    gate = randn(f, k, dtype=torch.bfloat16, seed=97, scale=0.1)
    up = randn(f, k, dtype=torch.bfloat16, seed=98, scale=0.1)
    mixed = torch.stack([gate.view(-1, 16, k), up.view(-1, 16, k)], dim=1).reshape(2 * f, k).contiguous()
    assert ops().glu_fusable(2 * f, k, torch.bfloat16)
    got = ops().linear(a, mixed, glu=True)
    g, u = a.float() @ gate.float().T, a.float() @ up.float().T
    want = g / (1 + torch.exp(-g)) * u
    assert got.shape == (m, f)
    assert torch.allclose(got.float(), want, atol=2e-2 * float(want.abs().max()), rtol=2e-2)
    assert torch.allclose(plain_ops.linear(a, mixed, glu=True).float(), want, atol=1e-2 * float(want.abs().max()), rtol=2e-2)
    assert ops().tensor_core_status() == 0


@pytest.mark.parametrize("m,n,k,cut", [(350, 4096, 4096, 0), (129, 2048, 14336, 0), (257, 2048, 8192, 0), (1300, 4096, 4096, 0),
                                       (300, 2112, 2056, 0), (777, 28672, 1024, 0), (2077, 6144, 1600, 0),
                                       (1153, 4128, 8200, 11), (1501, 9632, 4096, 6), (1501, 4120, 9608, 28), (2077, 6152, 4104, 3),
                                       (2077, 2080, 8192, 7), (3001, 2080, 8192, 34)])
def test_linear_cuts_the_last_round_of_tiles(m, n, k, cut):
    """Products whose last round of 256 x 256 tiles leaves pairs idle: its `cut` tiles are cut along K over all pairs and their
    parts added, for each epilogue, with one part order (two runs give the same bits); a few tiles in many parts and many in
    few, tokens and outputs that end inside a tile. With 0, shapes around them that other kernels take. Largest error of a sum of
    k products of bfloat16 values in 32 bits: k 2^-24 of the sum of magnitudes, far inside 2e-3 of the largest result."""
    assert not cut or all(ops().product_plan(m, n, k, target).tail == cut for target in ops().TARGETS)
    a = randn(m, k, dtype=torch.bfloat16, seed=201)
    w = randn(n, k, dtype=torch.bfloat16, seed=202, scale=0.05)
    bias = randn(n, seed=203)
    plain = a.double() @ w.double().T
    want = plain + bias.double()
    scale = float(want.abs().max())
    got = ops().linear(a, w, bias, out_dtype=torch.float32)
    assert float((got - want).abs().max()) <= 2e-3 * scale
    assert torch.equal(got, ops().linear(a, w, bias, out_dtype=torch.float32))
    assert float((ops().linear(a, w, bias).double() - want).abs().max()) <= 1e-2 * scale
    residual = randn(m, n, seed=204)
    expect = residual.double() + want
    ops().linear(a, w, bias, residual=residual)
    assert float((residual - expect).abs().max()) <= 2e-3 * scale
    if cut:
        norm = ops().FoldedNorm(a, _sums_in_parts(a, 3, 205), 3, 1e-5, k)
        rstd = 1.0 / torch.sqrt((a.double() ** 2).mean(dim=1, keepdim=True) + 1e-5)
        got = ops().linear(a, w, bias, out_dtype=torch.float32, norm=norm)
        assert float((got.double() - (plain * rstd + bias.double())).abs().max()) <= 2e-3 * scale
    if n % 32 == 0:
        f = n // 2
        gate, up = plain.view(m, f // 16, 2, 16).unbind(2)
        act = (gate / (1 + torch.exp(-gate)) * up).reshape(m, f)
        assert float((ops().linear(a, w, glu=True).double() - act).abs().max()) <= 1e-2 * float(act.abs().max())
    assert ops().tensor_core_status() == 0


@pytest.mark.parametrize("m,n,k", [(353, 6152, 1032), (350, 4102, 2056), (511, 4104, 4096), (256, 4104, 8192), (300, 4096, 4096),
                                   (190, 4096, 8192), (129, 6144, 4096), (1300, 4096, 1536), (140, 8224, 4104), (511, 4128, 4096),
                                   (300, 8224, 4104), (350, 12320, 2056), (400, 4096, 14336), (300, 28704, 2056), (1150, 12320, 1544)])
def test_linear_with_the_weights_on_the_row_side(m, n, k):
    """Products whose weights are the rows of the pairs' tiles: token tiles of several widths that end inside a tile and inside 16
    tokens, outputs that end inside a tile and a block, rows no tensor map can describe (4,102), K that ends inside a
    k-block, one pair a tile, up to six tiles a pair one after the other, and two or three pairs in a cluster; every epilogue, with a
    folded norm and without, the next norm's input behind the residual, one order of the sums (two runs give the same bits).
    Errors as in the test above; a square sum of n terms in 32 bits is off by n 2^-24 at most."""
    plans = {target: ops().product_plan(m, n, k, target) for target in ops().TARGETS}
    assert plans["float32"].kernel == plans["residual"].kernel == "row_side"
    a = randn(m, k, dtype=torch.bfloat16, seed=231)
    w = randn(n, k, dtype=torch.bfloat16, seed=232, scale=0.05)
    bias = randn(n, seed=233)
    plain = a.double() @ w.double().T
    want = plain + bias.double()
    scale = float(want.abs().max())
    got = ops().linear(a, w, bias, out_dtype=torch.float32)
    assert float((got - want).abs().max()) <= 2e-3 * scale
    assert torch.equal(got, ops().linear(a, w, bias, out_dtype=torch.float32))
    assert float((ops().linear(a, w, bias).double() - want).abs().max()) <= 1e-2 * scale
    residual = randn(m, n, seed=234)
    expect = residual.double() + want
    ops().linear(a, w, bias, residual=residual)
    assert float((residual - expect).abs().max()) <= 2e-3 * scale
    again = randn(m, n, seed=234)
    emit = _emit(m, n)
    ops().linear(a, w, bias, residual=again, emit=emit)
    assert torch.equal(again, residual) and torch.equal(emit.rows, residual.to(torch.bfloat16))
    squares = (residual.double() ** 2).sum(dim=1)
    assert float((emit.sumsq[:, :emit.parts].double().sum(dim=1) / squares - 1).abs().max()) <= n * 2.0 ** -24
    norm = ops().FoldedNorm(a, _sums_in_parts(a, 5, 235), 5, 1e-5, k)
    rstd = 1.0 / torch.sqrt((a.double() ** 2).mean(dim=1, keepdim=True) + 1e-5)
    assert float((ops().linear(a, w, bias, norm=norm).double() - (plain * rstd + bias.double())).abs().max()) <= 1e-2 * scale
    if n % 32 == 0:
        for scaled, kind, extra in ((plain, True, {}), (plain * rstd, "gelu", {"norm": norm})):
            gate, up = scaled.view(m, n // 32, 2, 16).unbind(2)
            act = gate / (1 + torch.exp(-gate)) if kind is True else torch.nn.functional.gelu(gate, approximate="tanh")
            act = (act * up).reshape(m, n // 2)
            assert float((ops().linear(a, w, glu=kind, **extra).double() - act).abs().max()) <= 1e-2 * float(act.abs().max())
    assert ops().tensor_core_status() == 0


@pytest.mark.parametrize("m,n,k,kernel", [(350, 4096, 4096, "row_side"), (1153, 4128, 8200, "pairs"), (200, 2048, 4096, "blocks")])
def test_linear_on_two_streams_at_once(m, n, k, kernel):
    """Products on two streams with nothing between them, where the kernel leaves parts in scratch (tiles cut along K, split K) and
    where it needs none: each stream has its own."""
    plan = ops().product_plan(m, n, k)
    assert plan.kernel == kernel and (plan.scratch_floats > 0) == (kernel != "row_side")
    a = randn(m, k, dtype=torch.bfloat16, seed=205)
    ws = [randn(n, k, dtype=torch.bfloat16, seed=206 + i, scale=0.05) for i in range(2)]
    want = [ops().linear(a, w) for w in ws]
    streams = [torch.cuda.Stream() for _ in ws]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(10):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                got[i].append(ops().linear(a, ws[i]))
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i]) for i in range(2) for g in got[i])


@pytest.mark.parametrize("m,n,k", [(350, 4096, 4096), (64, 4096, 4096), (1153, 4128, 8200)])      # sums in a cluster; K split over blocks; parts of tiles
def test_products_on_many_streams_and_in_a_graph_at_once(m, n, k):
    """More streams than keep scratch, and a captured product replayed on one more, with nothing between them: the bits of
    single calls."""
    a = randn(m, k, dtype=torch.bfloat16, seed=211)
    ws = [randn(n, k, dtype=torch.bfloat16, seed=212 + i, scale=0.05) for i in range(3)]
    want = [ops().linear(a, w) for w in ws]
    streams = [torch.cuda.Stream() for _ in range(11)]
    graphs, captured = [], []
    for w in ws[:2]:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured.append([ops().linear(a, w), ops().linear(a, ws[2])])
        graphs.append(graph)
    torch.cuda.synchronize()
    got = []
    for turn in range(5):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                if i in (3, 7):
                    graphs[i == 7].replay()
                else:
                    got.append((i % 3, ops().linear(a, ws[i % 3])))
        if turn < 4:
            continue
        torch.cuda.synchronize()
    assert all(torch.equal(g, want[w]) for w, g in got)
    assert all(torch.equal(c[0], want[i]) and torch.equal(c[1], want[2]) for i, c in enumerate(captured))
    assert ops().tensor_core_status() == 0


def test_two_engines_on_two_streams_at_once():
    """Prompts, recorded passes and replayed decode steps of two engines, each on its stream with nothing between them: the
    logits of the same steps alone."""
    from llm_b200.config import config_from_dict
    from llm_b200.engine import DecoderModel, Engine, Entry
    from llm_b200.shapes import shape
    config = config_from_dict(shape("llama-3.2-1b", 2))

    def engine(seed):
        gen = torch.Generator(device=DEV).manual_seed(seed)
        model = DecoderModel(config.model_spec())
        weights = {name: torch.empty(spec.shape, dtype=torch.bfloat16, device=DEV).normal_(generator=gen).mul_(0.02)
                   for name, spec in model.parameters().items()}
        model.bind(weights, torch.bfloat16, DEV)
        return Engine(model, max_tokens=2048, max_seq_len=512, max_slots=4)

    def steps(e, seed):
        """A generator of logits: three prompts of one size (plain, recorded, run from the record), then decode steps."""
        gen = torch.Generator().manual_seed(seed)
        ids = lambda n: torch.randint(0, 1000, (n,), generator=gen).tolist()      # noqa: E731
        for _ in range(3):
            slots = e.acquire(1)
            yield e.step([Entry(slots[0], ids(300), [299])])
            e.release(slots)
        slots = e.acquire(2)
        yield e.step([Entry(s, ids(200), [199]) for s in slots])
        for _ in range(6):
            yield e.step([Entry(s, ids(1), [0]) for s in slots])

    engines = [engine(seed) for seed in (1, 2)]
    alone = []
    for i in (0, 1):
        alone.append([logits.clone() for logits in steps(engine(i + 1), 7 + i)])
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in engines]
    torch.cuda.synchronize()
    runs, both = [steps(e, 7 + i) for i, e in enumerate(engines)], [[], []]
    for _ in alone[0]:
        for i in (0, 1):
            with torch.cuda.stream(streams[i]):
                both[i].append(next(runs[i]))
    torch.cuda.synchronize()
    assert all(e.records_run >= 1 and e.graph_replays >= 1 for e in engines)
    for i in (0, 1):
        assert all(torch.equal(x, y) for x, y in zip(alone[i], both[i])), i


def test_linear_rows_do_not_depend_on_the_batch():
    """32-bit: a row's product is bit-equal whether it is computed alone or among 200 rows."""
    a = randn(200, 172, seed=8)
    w = randn(300, 172, seed=9)
    whole = ops().linear(a, w)
    for row in (0, 63, 64, 199):
        assert torch.equal(ops().linear(a[row:row + 1].contiguous(), w)[0], whole[row])


def make_cache(n_seqs, lens, n_kv_heads, head_dim, dtype, seed, ring_pages=None):
    """A shuffled page pool, block tables, and keys/values written position by position."""
    width = ring_pages or max((n + 63) // 64 for n in lens) + 1
    n_pages = n_seqs * width + 3
    gen = torch.Generator().manual_seed(seed)
    perm = torch.randperm(n_pages, generator=gen)
    table = perm[:n_seqs * width].view(n_seqs, width).to(torch.int32).to(DEV)
    k_cache = torch.full((n_pages, n_kv_heads, 64, head_dim), 7.0, dtype=dtype, device=DEV)
    v_cache = torch.full((n_pages, n_kv_heads, 64, head_dim), -9.0, dtype=dtype, device=DEV)
    return table, width, k_cache, v_cache


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,dim,interleaved", [(4, 2, 16, False), (3, 1, 32, True),
                                                            (8, 8, 64, False), (16, 2, 128, False),
                                                            (2, 1, 256, False), (6, 2, 48, False)])
def test_rope_cache_write(dtype, heads, kv_heads, dim, interleaved):
    starts, counts = [0, 70, 5], [9, 1, 130]
    lens = [s + c for s, c in zip(starts, counts)]
    table, width, k_cache, v_cache = make_cache(3, lens, kv_heads, dim, dtype, 10)
    tok_pos = torch.tensor([p for s, c in zip(starts, counts) for p in range(s, s + c)],
                           dtype=torch.int32, device=DEV)
    tok_seq = torch.tensor([b for b, c in enumerate(counts) for _ in range(c)],
                           dtype=torch.int32, device=DEV)
    n = tok_pos.numel()
    qkv = randn(n, (heads + 2 * kv_heads) * dim, dtype=dtype, seed=11)
    angle = torch.arange(256, dtype=torch.float64)[:, None] * (
        10000.0 ** (-2.0 * torch.arange(dim // 2, dtype=torch.float64) / dim))[None, :]
    rope = torch.cat([angle.cos(), angle.sin()], 1).float().to(DEV)
    expect_qkv, expect_k, expect_v = qkv.clone(), k_cache.clone(), v_cache.clone()
    plain_ops.rope_cache_write(expect_qkv, rope, tok_pos, tok_seq, table, width, expect_k,
                               expect_v, heads, kv_heads, dim, interleaved)
    ops().rope_cache_write(qkv, rope, tok_pos, tok_seq, table, width, k_cache, v_cache, heads,
                           kv_heads, dim, interleaved)
    t = tol(dtype)
    assert torch.allclose(qkv.float(), expect_qkv.float(), **t)
    assert torch.allclose(k_cache.float(), expect_k.float(), **t)     # untouched rows keep 7.0
    assert torch.allclose(v_cache.float(), expect_v.float(), **t)
    # without a table nothing turns; without write_cache the cache stays
    q2, k2, v2 = qkv.clone(), k_cache.clone(), v_cache.clone()
    ops().rope_cache_write(q2, None, tok_pos, tok_seq, table, width, k2, v2, heads, kv_heads, dim,
                           interleaved, write_cache=False)
    assert torch.equal(q2, qkv) and torch.equal(k2, k_cache) and torch.equal(v2, v_cache)


def fill_cache(table, width, k_cache, v_cache, lens, seed):
    """Random keys and values at every position < len of every sequence."""
    kv_heads, dim = k_cache.shape[1], k_cache.shape[3]
    keys, values = [], []
    for b, n in enumerate(lens):
        k = randn(n, kv_heads, dim, seed=seed + 2 * b)
        v = randn(n, kv_heads, dim, seed=seed + 2 * b + 1)
        pos = torch.arange(n, device=DEV)
        pages = table[b].long()[(pos // 64) % width]
        k_cache[pages, :, pos % 64, :] = k.to(k_cache.dtype)
        v_cache[pages, :, pos % 64, :] = v.to(v_cache.dtype)
        keys.append(k)
        values.append(v)
    return keys, values


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,dim,window", [(4, 2, 16, 0), (3, 1, 32, 0), (8, 1, 64, 0),
                                                       (8, 2, 128, 0), (2, 2, 256, 0),
                                                       (6, 2, 48, 0), (4, 2, 32, 37)])
def test_attention_prefill_and_decode(dtype, heads, kv_heads, dim, window):
    lens = [130, 1, 77, 300]
    table, width, k_cache, v_cache = make_cache(4, lens, kv_heads, dim, dtype, 20)
    fill_cache(table, width, k_cache, v_cache, lens, 21)
    scale = 1.0 / math.sqrt(dim)
    # prefill: every position of every sequence is a query
    tok_pos = torch.tensor([p for n in lens for p in range(n)], dtype=torch.int32, device=DEV)
    tok_seq = torch.tensor([b for b, n in enumerate(lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    qkv = randn(tok_pos.numel(), (heads + 2 * kv_heads) * dim, dtype=dtype, seed=22)
    got = ops().attention(qkv, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads,
                          dim, scale, window)
    want = plain_ops.attention(qkv, k_cache, v_cache, table, width, tok_pos, tok_seq, heads,
                               kv_heads, dim, scale, window)
    assert torch.allclose(got.float(), want.float(), **tol(dtype))
    # decode: one query per sequence at its last position
    last = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    seqs = torch.arange(4, dtype=torch.int32, device=DEV)
    q1 = randn(4, (heads + 2 * kv_heads) * dim, dtype=dtype, seed=23)
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got = ops().attention(q1, k_cache, v_cache, table, width, last, seqs, heads, kv_heads, dim,
                          scale, window, decode=True, seq_lens=seq_lens, max_len=max(lens))
    want = plain_ops.attention(q1, k_cache, v_cache, table, width, last, seqs, heads, kv_heads,
                               dim, scale, window)
    assert torch.allclose(got.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("heads,kv_heads,dim", [(32, 8, 128), (8, 1, 64), (6, 2, 96), (4, 4, 32),
                                                (3, 1, 128)])
@pytest.mark.parametrize("forced_slices", [0, 1, 2, 16])
def test_attention_decode_kernel_long_contexts(heads, kv_heads, dim, forced_slices, monkeypatch):
    """The split-KV decode kernel at lengths from 1 to 3000 in one batch (page edges,
    empty slices, many slices), twice in a row on the same scratch; with the library's own
    choice of slices and with forced counts (one slice writes the result without the
    combining kernel)."""
    if forced_slices:
        monkeypatch.setenv("LLMB_DECODE_SPLITS", str(forced_slices))
    from llm_b200.ops import tactics
    dtype = torch.bfloat16
    assert tactics.choose_attention(True, dtype, heads, kv_heads, dim, 0) == "attention_decode"
    lens = [3000, 1, 64, 65, 1000, 127]
    table, width, k_cache, v_cache = make_cache(len(lens), lens, kv_heads, dim, dtype, 90)
    fill_cache(table, width, k_cache, v_cache, lens, 91)
    last = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    seqs = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    q = randn(len(lens), (heads + 2 * kv_heads) * dim, dtype=dtype, seed=92)
    want = plain_ops.attention(q, k_cache, v_cache, table, width, last, seqs, heads, kv_heads, dim,
                               dim ** -0.5)
    longest_first = torch.tensor(sorted(range(len(lens)), key=lambda b: -lens[b]), dtype=torch.int32, device=DEV)
    for order in (None, longest_first):          # the second call also takes the sequences longest first
        got = ops().attention(q, k_cache, v_cache, table, width, last, seqs, heads, kv_heads, dim,
                              dim ** -0.5, 0, decode=True, seq_lens=seq_lens, max_len=max(lens),
                              seq_order=order)
        assert torch.allclose(got.float(), want.float(), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (4, 1, 64), (6, 2, 96), (4, 4, 32),
                                                (3, 1, 128)])
@pytest.mark.parametrize("variant", ["attention_prefill", "attention_prefill_tc"])
def test_attention_prefill_kernel(heads, kv_heads, dim, variant):
    """The flash prefill kernels (mma.sync and tcgen05): sequences that start at position 0
    and sequences that continue (chunked prompts), lengths around tile and page edges."""
    from llm_b200.ops import tactics
    if variant == "attention_prefill_tc" and dim not in (64, 128):
        pytest.skip("the tcgen05 kernel serves head sizes 64 and 128")
    if variant == "attention_prefill":
        tactics.disable("attention_prefill_tc")
    try:
        assert tactics.choose_attention(False, torch.bfloat16, heads, kv_heads, dim, 0, True) == variant
        _check_prefill_attention(heads, kv_heads, dim)
        ops().check_device_status()
    finally:
        tactics.enable("attention_prefill_tc")


def _check_prefill_attention(heads, kv_heads, dim):
    dtype = torch.bfloat16
    starts, counts = [0, 0, 100, 64, 0, 300], [300, 1, 65, 64, 63, 130]
    lens = [s + c for s, c in zip(starts, counts)]
    table, width, k_cache, v_cache = make_cache(len(lens), lens, kv_heads, dim, dtype, 93)
    fill_cache(table, width, k_cache, v_cache, lens, 94)
    tok_pos = torch.tensor([p for s, c in zip(starts, counts) for p in range(s, s + c)],
                           dtype=torch.int32, device=DEV)
    tok_seq = torch.tensor([b for b, c in enumerate(counts) for _ in range(c)], dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=DEV)
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    q = randn(tok_pos.numel(), (heads + 2 * kv_heads) * dim, dtype=dtype, seed=95)
    want = plain_ops.attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads,
                               dim, dim ** -0.5)
    longest_first = torch.tensor(sorted(range(len(lens)), key=lambda b: -lens[b]), dtype=torch.int32, device=DEV)
    for order in (None, longest_first):
        got = ops().attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads, dim,
                              dim ** -0.5, 0, seq_lens=seq_lens, max_len=max(lens), cu_seqlens=cu,
                              max_new=max(counts), seq_order=order)
        assert torch.allclose(got.float(), want.float(), atol=2e-2, rtol=2e-2)
        # and relative to each row's norm: random softmax outputs are small, a lost key must show
        g, w = got.float().view(-1, heads, dim), want.float().view(-1, heads, dim)
        relative = (g - w).norm(dim=-1) / w.norm(dim=-1).clamp_min(1e-3)
        assert float(relative.max()) < 0.03


@pytest.mark.parametrize("variant", ["attention_prefill", "attention_prefill_tc"])
@pytest.mark.parametrize("dim", [64, 128])
def test_attention_prefill_growing_scores(variant, dim):
    """Keys grow from one block of 128 to the next, first a little and then by much, so that a
    row's running maximum moves late in the sequence: by less than the kernel's threshold for
    rescaling (probabilities above one) and by far more (the accumulated output is rescaled)."""
    from llm_b200.ops import tactics
    heads, kv_heads, dtype, n = 4, 2, torch.bfloat16, 700
    if variant == "attention_prefill":
        tactics.disable("attention_prefill_tc")
    try:
        assert tactics.choose_attention(False, dtype, heads, kv_heads, dim, 0, True) == variant
        table, width, k_cache, v_cache = make_cache(1, [n], kv_heads, dim, dtype, 96)
        fill_cache(table, width, k_cache, v_cache, [n], 97)
        for block, factor in enumerate([0.3, 1.0, 1.4, 0.5, 6.0, 2.0]):
            for page in (2 * block, 2 * block + 1):
                if page < width:
                    k_cache[int(table[0, page])] *= factor
        tok_pos = torch.arange(n, dtype=torch.int32, device=DEV)
        tok_seq = torch.zeros(n, dtype=torch.int32, device=DEV)
        cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
        seq_lens = torch.tensor([n], dtype=torch.int32, device=DEV)
        q = randn(n, (heads + 2 * kv_heads) * dim, dtype=dtype, seed=98)
        want = plain_ops.attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads,
                                   dim, dim ** -0.5)
        got = ops().attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads, dim,
                              dim ** -0.5, 0, seq_lens=seq_lens, max_len=n, cu_seqlens=cu, max_new=n)
        assert torch.allclose(got.float(), want.float(), atol=2e-2, rtol=2e-2)
        ops().check_device_status()
    finally:
        tactics.enable("attention_prefill_tc")


@pytest.mark.parametrize("variant", ["attention_prefill", "attention_prefill_tc"])
@pytest.mark.parametrize("start,count", [(173, 2), (173, 129), (100, 130), (0, 300)])
def test_prefill_attention_finds_planted_keys(variant, start, count):
    """Random scores over hundreds of keys hide one lost or wrongly masked key, so keys are
    planted: one early key (position 3), the key just before a continued chunk's first token,
    and the chunk's last key. A query that points at a planted key must return that key's value
    (a query in the chunk's last tile, a chunk that starts off the tile and page edges); the query
    one position before the last key must not see it."""
    from llm_b200.ops import tactics
    heads, kv_heads, dim, dtype = 4, 2, 128, torch.bfloat16
    n = start + count
    if variant == "attention_prefill":
        tactics.disable("attention_prefill_tc")
    try:
        assert tactics.choose_attention(False, dtype, heads, kv_heads, dim, 0, True) == variant
        direction = torch.zeros(dim, device=DEV)
        direction[5] = 40.0
        tok_pos = torch.arange(start, n, dtype=torch.int32, device=DEV)
        tok_seq = torch.zeros(count, dtype=torch.int32, device=DEV)
        cu = torch.tensor([0, count], dtype=torch.int32, device=DEV)
        seq_lens = torch.tensor([n], dtype=torch.int32, device=DEV)
        cases = [(3, n - 1, True), (n - 1, n - 1, True)]
        if start > 0:
            cases += [(start - 1, start, True), (start - 1, n - 1, True)]
        if count >= 2:
            cases += [(n - 1, n - 2, False)]
        for key_pos, query_pos, seen in cases:
            table, width, k_cache, v_cache = make_cache(1, [n], kv_heads, dim, dtype, 130)
            keys, values = fill_cache(table, width, k_cache, v_cache, [n], 131)
            k_cache[int(table[0, key_pos // 64]), :, key_pos % 64, :] = direction.to(dtype)
            q = randn(count, (heads + 2 * kv_heads) * dim, dtype=dtype, seed=132, scale=0.1)
            q[query_pos - start, :heads * dim] = direction.repeat(heads).to(dtype)
            got = ops().attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads, dim,
                                  dim ** -0.5, 0, seq_lens=seq_lens, max_len=n, cu_seqlens=cu, max_new=count)
            row = got[query_pos - start].float().view(heads, dim)
            for h in range(heads):
                expect = values[0][key_pos, h // 2].to(dtype).float()
                hit = torch.allclose(row[h], expect, atol=2e-2)
                assert hit == seen, (key_pos, query_pos, h)
        ops().check_device_status()
    finally:
        tactics.enable("attention_prefill_tc")


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_finds_one_far_key(dtype):
    """Among 500 keys one early key matches the query; the output must be its
    value, and with a window that excludes it, must not be."""
    heads, kv_heads, dim, n = 4, 2, 64, 500
    table, width, k_cache, v_cache = make_cache(1, [n], kv_heads, dim, dtype, 30)
    keys, values = fill_cache(table, width, k_cache, v_cache, [n], 31)
    far = 3
    direction = torch.zeros(dim, device=DEV)
    direction[5] = 40.0
    page = int(table[0, far // 64])
    k_cache[page, :, far % 64, :] = direction.to(dtype)
    qkv = torch.zeros(1, (heads + 2 * kv_heads) * dim, dtype=dtype, device=DEV)
    qkv[0, :heads * dim] = direction.repeat(heads).to(dtype)
    pos = torch.tensor([n - 1], dtype=torch.int32, device=DEV)
    seq = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = ops().attention(qkv, k_cache, v_cache, table, width, pos, seq, heads, kv_heads, dim,
                          1.0 / math.sqrt(dim), 0, decode=True,
                          seq_lens=torch.tensor([n], dtype=torch.int32, device=DEV), max_len=n)
    got = got.float().view(heads, dim)
    for h in range(heads):
        expect = values[0][far, h // 2].to(dtype).float()
        assert torch.allclose(got[h], expect, atol=2e-2)
    windowed = ops().attention(qkv, k_cache, v_cache, table, width, pos, seq, heads, kv_heads,
                               dim, 1.0 / math.sqrt(dim), 100).float().view(heads, dim)
    assert not torch.allclose(windowed[0], values[0][far, 0].to(dtype).float(), atol=0.1)


@pytest.mark.usefixtures("prefill_form")
@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 2, 128), (4, 4, 64), (32, 1, 128)])
@pytest.mark.parametrize("window", [1, 64, 130, 300])
@pytest.mark.parametrize("extras", [False, True])
def test_windowed_prefill_on_tcgen05(heads, kv_heads, dim, window, extras):
    """Windows that begin inside a key block, blocks that only some rows of a tile see, with a sink, a gate and a scale."""
    starts, counts = [0, 700, 63, 0], [300, 257, 1, 128]
    lens = [s + c for s, c in zip(starts, counts)]
    table, width, k_cache, v_cache = make_cache(4, lens, kv_heads, dim, torch.bfloat16, 96)
    fill_cache(table, width, k_cache, v_cache, lens, 97)
    tok_pos = torch.tensor([p for s, c in zip(starts, counts) for p in range(s, s + c)], dtype=torch.int32, device=DEV)
    tok_seq = torch.tensor([b for b, c in enumerate(counts) for _ in range(c)], dtype=torch.int32, device=DEV)
    cu = torch.tensor([sum(counts[:i]) for i in range(5)], dtype=torch.int32, device=DEV)
    seq_lens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    n = tok_pos.numel()
    q = randn(n, heads * dim, dtype=torch.bfloat16, seed=98)
    more = dict(sinks=randn(heads, seed=99), gate=randn(n, heads, dtype=torch.bfloat16, seed=100), out_scale=0.7) if extras else {}
    want = plain_ops.attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads, dim, dim ** -0.5, window, **more)
    got = ops().attention(q, k_cache, v_cache, table, width, tok_pos, tok_seq, heads, kv_heads, dim, dim ** -0.5, window,
                          seq_lens=seq_lens, max_len=max(lens), cu_seqlens=cu, max_new=max(counts), **more)
    ops().check_device_status()
    assert torch.allclose(got.float(), want.float(), atol=2e-2, rtol=2e-2)
    g, w = got.float().view(-1, heads, dim), want.float().view(-1, heads, dim)
    assert float(((g - w).norm(dim=-1) / w.norm(dim=-1).clamp_min(1e-3)).max()) < 0.03


def test_attention_window_edge():
    """The key at position p - window is out, the key at p - window + 1 is in."""
    heads, kv_heads, dim, n, window = 2, 1, 32, 200, 64
    dtype = torch.float32
    table, width, k_cache, v_cache = make_cache(1, [n], kv_heads, dim, dtype, 40)
    keys, values = fill_cache(table, width, k_cache, v_cache, [n], 41)
    direction = torch.zeros(dim, device=DEV)
    direction[0] = 50.0
    qkv = torch.zeros(1, (heads + 2) * dim, device=DEV)
    qkv[0, :heads * dim] = direction.repeat(heads)
    pos = torch.tensor([n - 1], dtype=torch.int32, device=DEV)
    seq = torch.zeros(1, dtype=torch.int32, device=DEV)
    for key_pos, inside in ((n - 1 - window, False), (n - window, True)):
        kc = k_cache.clone()
        kc[int(table[0, key_pos // 64]), :, key_pos % 64, :] = direction
        got = ops().attention(qkv, kc, v_cache, table, width, pos, seq, heads, kv_heads, dim,
                              1.0 / math.sqrt(dim), window).view(heads, dim)
        hit = torch.allclose(got[0], values[0][key_pos, 0], atol=1e-3)
        assert hit == inside


def test_argmax_first_maximum_wins():
    logits = randn(5, 1000, seed=50)
    logits[1, 700] = logits[1, 20] = 9.0
    logits[2] = 0.0
    got = ops().argmax_rows(logits)
    assert got.tolist() == plain_ops.argmax_rows(logits).tolist()
    assert got[1] == 20 and got[2] == 0


def _sampler_state(n, params, iparams, seeds, cap=8):
    f = torch.tensor(params, dtype=torch.float32, device=DEV)
    i = torch.tensor(iparams, dtype=torch.int32, device=DEV)
    rng = torch.tensor([(s | 1) - (1 << 64) if (s | 1) >= (1 << 63) else (s | 1) for s in seeds],
                       dtype=torch.int64, device=DEV)
    recent = torch.zeros((n, cap), dtype=torch.int32, device=DEV)
    recent_len = torch.zeros((n,), dtype=torch.int32, device=DEV)
    out = torch.zeros((n,), dtype=torch.int32, device=DEV)
    status = torch.zeros((n,), dtype=torch.int32, device=DEV)
    return f, i, recent, recent_len, rng, out, status


@pytest.mark.parametrize("vocab", [384, 5000, 50001])
def test_sample_rows_matches_plain_chain(vocab):
    """Greedy, temperature with top-k / top-p / min-p, penalty, and no top-k at all:
    the same tokens and generator states as the plain chain, over several draws. 50,001 entries:
    rows that are read four values a load, eight loads ahead, with a tail that is not."""
    params = [[0.0, 0.75, 0.25, 1.0], [0.8, 0.75, 0.25, 1.1], [1.5, 0.95, 0.0, 1.3],
              [1.0, 1.0, 0.0, 1.0], [0.7, 2.0, 0.05, 1.0]]
    iparams = [[40, 64], [40, 64], [7, 4], [0, 0], [0, 0]]
    seeds = [1, 1, 0x5EED1234ABCD0001, 99, 12345]
    n = len(params)
    state_gpu = _sampler_state(n, params, iparams, seeds)
    state_cpu = [t.cpu().clone() for t in state_gpu]
    state_gpu[2][:, :3] = torch.tensor([3, 3, 10], dtype=torch.int32)
    state_cpu[2][:, :3] = torch.tensor([3, 3, 10], dtype=torch.int32)
    state_gpu[3][:] = 3
    state_cpu[3][:] = 3
    for draw in range(6):
        logits = randn(n, vocab, seed=60 + draw, scale=2.5)
        logits[:, 3] = 4.0            # a penalised token that matters
        cpu_logits = logits.cpu().clone()
        ops().sample_rows(logits, *state_gpu)
        plain_ops.sample_rows(cpu_logits, *state_cpu)
        assert state_gpu[5].tolist() == state_cpu[5].tolist(), f"draw {draw}"
        assert state_gpu[4].tolist() == state_cpu[4].tolist()
        assert state_gpu[6].tolist() == [0] * n


def test_sample_rows_records_windows_and_finds_state_by_row():
    """Three logits rows that belong to sequences 4, 0 and 2 of a batch of five: the kernel takes each
    row's parameters, window and generator from its sequence's row, enters the drawn token into that
    window, and leaves the other sequences' state alone; three draws in a row against the plain chain."""
    vocab, n = 777, 5
    params = [[0.9, 0.9, 0.05, 1.2]] * n
    iparams = [[30, 6]] * n
    state_gpu = _sampler_state(n, params, iparams, [11, 12, 13, 14, 15], cap=6)
    state_cpu = [t.cpu().clone() for t in state_gpu]
    rows = torch.tensor([4, 0, 2], dtype=torch.int32)
    out_gpu, out_cpu = torch.zeros(3, dtype=torch.int32, device=DEV), torch.zeros(3, dtype=torch.int32)
    for draw in range(8):                               # more draws than the window holds
        logits = randn(3, vocab, seed=200 + draw, scale=2.0)
        cpu_logits = logits.cpu().clone()
        f, i, recent, recent_len, rng, _, status = state_gpu
        ops().sample_rows(logits, f, i, recent, recent_len, rng, out_gpu, status, record=True,
                          state_rows=rows.to(DEV))
        f, i, recent, recent_len, rng, _, status = state_cpu
        plain_ops.sample_rows(cpu_logits, f, i, recent, recent_len, rng, out_cpu, status, record=True,
                              state_rows=rows)
        assert out_gpu.tolist() == out_cpu.tolist(), draw
        for g, c in zip(state_gpu[2:5], state_cpu[2:5]):
            assert g.tolist() == c.tolist(), draw
    assert state_gpu[3].tolist() == [8, 0, 8, 0, 8]


def test_sample_rows_refuses_what_it_cannot_rank():
    f, i, recent, recent_len, rng, out, status = _sampler_state(
        2, [[1.0, 0.9, 0.0, 1.0], [1.0, 1.0, 0.0, 1.0]], [[0, 0], [2000, 0]], [1, 2])
    logits = randn(2, 5000, seed=70)
    ops().sample_rows(logits, f, i, recent, recent_len, rng, out, status)
    assert status.tolist() == [1, 1]


def test_a_refused_row_stays_flagged_over_later_steps():
    """4,096 equal logits at a top-k cut of 40 are more ties than the kernel ranks: the row is refused.
    The next launch, on logits it can rank, must not erase the flag (only the host clears it)."""
    f, i, recent, recent_len, rng, out, status = _sampler_state(
        2, [[1.0, 0.9, 0.0, 1.0], [1.0, 0.9, 0.0, 1.0]], [[40, 0], [40, 0]], [1, 2])
    logits = torch.zeros(2, 4096, device=DEV)
    logits[1] = randn(1, 4096, seed=71)[0]
    ops().sample_rows(logits, f, i, recent, recent_len, rng, out, status)
    assert status.tolist() == [1, 0] and out.tolist()[0] == 0
    ops().sample_rows(randn(2, 4096, seed=72), f, i, recent, recent_len, rng, out, status)
    assert status.tolist() == [1, 0]


@pytest.mark.parametrize("vocab", [1, 5, 31, 1024, 1025, 4097, 32003, 128256])
@pytest.mark.parametrize("steps", [0, 3, 60])
def test_sample_rows_over_a_cluster(vocab, steps):
    """Rows shared by the blocks of a cluster: shares that are empty, end inside four entries or differ in
    size; continuous logits (the select ends after one digit) and logits on a grid of `steps` values (runs of
    equal ones at the cut, more of them in a bin than the candidate buffer holds): tokens, windows and generators
    of the plain chain, or refused together with it."""
    n = 4
    top = min(vocab, 40)
    params = [[0.7, 0.75, 0.25, 1.1], [1.0, 0.9, 0.0, 1.0], [0.0, 0.75, 0.25, 1.2], [1.3, 2.0, 0.1, 1.0]]
    iparams = [[top if top < vocab else 0, 8], [1, 0], [0, 8], [min(1024, max(vocab - 1, 1)), 0]]
    state_gpu = _sampler_state(n, params, iparams, [3, 4, 5, 6])
    state_cpu = [t.cpu().clone() for t in state_gpu]
    for draw in range(3):
        logits = randn(n, vocab, seed=300 + draw, scale=2.0)
        if steps:
            logits = torch.round(logits * steps) / steps
        ranked = [v if 0 < v[0] < vocab or vocab <= 1024 else None for v in iparams]
        ties = [ranked[r] is not None and params[r][0] > 0 and iparams[r][0] > 0
                and int((logits[r] >= torch.topk(logits[r], min(iparams[r][0], vocab)).values[-1]).sum()) > 2048 for r in range(n)]
        cpu_logits = logits.cpu().clone()
        ops().sample_rows(logits, *state_gpu, record=True)
        plain_ops.sample_rows(cpu_logits, *state_cpu, record=True)
        for r in range(n):
            if ties[r] or int(state_gpu[6][r]) != 0:
                assert int(state_gpu[6][r]) == 1 and (ties[r] or int(state_cpu[6][r]) == 1), (r, draw)
                for g, c in zip(state_gpu, state_cpu):           # the same state for the draws that follow
                    c[r] = g[r].cpu()
                continue
            assert int(state_gpu[5][r]) == int(state_cpu[5][r]), (r, draw)
            assert state_gpu[4][r] == state_cpu[4][r].to(DEV) and state_gpu[2][r].tolist() == state_cpu[2][r].tolist()


@pytest.mark.parametrize("allowed", [3, 39, 41, 700, 5000])
def test_sample_rows_of_mostly_masked_logits(allowed):
    """Rows that are -inf but for a few entries, all of them in one block's share or spread: the shares' own cuts then lie at
    -inf, and where that is all a row has, its select runs over the whole row (or is refused for its ties, as before)."""
    vocab, n = 128256, 4
    params = [[0.7, 0.75, 0.25, 1.1], [1.0, 0.9, 0.0, 1.0], [1.3, 2.0, 0.1, 1.0], [0.8, 0.95, 0.0, 1.0]]
    state_gpu = _sampler_state(n, params, [[40, 8], [1, 0], [600, 0], [40, 8]], [3, 4, 5, 6])
    state_cpu = [t.cpu().clone() for t in state_gpu]
    full = randn(n, vocab, seed=320, scale=2.0)
    places = torch.randperm(vocab, generator=torch.Generator().manual_seed(allowed))[:allowed]
    logits = torch.full_like(full, float("-inf"))
    logits[:2, :allowed] = full[:2, :allowed]
    logits[2:, places.to(DEV)] = full[2:, :allowed]
    cpu_logits = logits.cpu().clone()
    ops().sample_rows(logits, *state_gpu, record=True)
    plain_ops.sample_rows(cpu_logits, *state_cpu, record=True)
    for r, k in enumerate((40, 1, 600, 40)):
        if k > allowed:
            assert int(state_gpu[6][r]) == 1, r              # more than 2,048 equal ones at the cut
        else:
            assert int(state_gpu[6][r]) == 0 and int(state_gpu[5][r]) == int(state_cpu[5][r]), r
            assert state_gpu[4][r] == state_cpu[4][r].to(DEV), r


@pytest.mark.parametrize("rows,vocab", [(1, 1), (3, 7), (2, 33), (5, 4099), (33, 128256)])
def test_argmax_over_a_cluster(rows, vocab):
    """First maximum over the blocks' shares, also with equal maxima in several shares and rows of -inf and NaN."""
    x = randn(rows, vocab, seed=310)
    x[0] = float("-inf")
    if rows > 1:
        x[1, vocab // 2:] = 7.0                                   # equal maxima from there on
        x[1, 0] = float("nan")
    want = [0 if r == 0 else vocab // 2 if r == 1 else int(x[r].argmax()) for r in range(rows)]
    if rows > 1 and vocab // 2 == 0:
        want[1] = 0
    assert ops().argmax_rows(x).tolist() == want


@pytest.mark.parametrize("vocab", [2048, 14336, 16380, 16384, 18436, 30720, 32772])
def test_argmax_at_the_ends_of_rounds(vocab):
    """A block reads 16,384 entries a round, the last round's in pieces of 2,048: maxima at the first and last entry of either,
    alone and with an equal one behind."""
    ends = sorted({i for edge in range(0, vocab + 2048, 2048) for i in (edge - 1, edge, vocab - 1) if 0 <= i < vocab})
    x = randn(len(ends), vocab, seed=312).clamp_(max=5.0)
    for r, i in enumerate(ends):
        x[r, i] = 7.0
        if r % 2:
            x[r, ends[r:]] = 7.0
    assert ops().argmax_rows(x).tolist() == ends


@pytest.mark.parametrize("vocab,rows", [(384, 3), (5000, 3), (20000, 3), (20000, 40)])
def test_sample_the_first_of_equal_logits(vocab, rows):
    """top_k of one: the first of 1 to 1,500 equal maxima is drawn (fewer and more than a warp, than the threads of a block), the
    generator moves on as in the plain chain, and more equal ones than the candidates' room are refused."""
    state_gpu = _sampler_state(rows, [[0.7, 0.95, 0.05, 1.0]] * rows, [[1, 0]] * rows, list(range(3, 3 + rows)))
    state_cpu = [t.cpu().clone() for t in state_gpu]
    for equal in (1, 2, 33, 300, 1500, 2500):
        if equal >= vocab:
            continue
        logits = randn(rows, vocab, seed=340 + equal).clamp_(max=3.0)
        for r in range(rows):
            places = torch.randperm(vocab, generator=torch.Generator().manual_seed(equal + r))[:equal]
            logits[r, places.to(DEV)] = 4.0
        cpu_logits = logits.cpu().clone()
        before = state_gpu[4].clone()
        ops().sample_rows(logits, *state_gpu)
        if equal > 2048:
            assert state_gpu[6].tolist() == [1] * rows and torch.equal(state_gpu[4], before)
            continue
        plain_ops.sample_rows(cpu_logits, *state_cpu)
        assert state_gpu[5].tolist() == state_cpu[5].tolist(), equal
        assert state_gpu[4].tolist() == state_cpu[4].tolist()
        assert state_gpu[6].tolist() == [0] * rows


@pytest.mark.parametrize("n,k", [(16, 4), (17, 64), (64, 172), (344, 64), (1000, 68), (100, 4096), (4099, 260)])
@pytest.mark.parametrize("residual", [False, True])
def test_linear_of_few_rows_in_32_bit(n, k, residual):
    """Up to 8 rows run a kernel of their own: the bits of the tiled kernel for the same rows (9 of them), for every
    number of rows, with edges in the columns, in the last tile of k, and a bias."""
    x, w, b = randn(9, k, seed=320), randn(n, k, seed=321), randn(n, seed=322)
    start = randn(9, n, seed=323)

    def run(m):
        if residual:
            acc = start[:m].clone()
            ops().linear(x[:m], w, b, residual=acc)
            return acc
        return ops().linear(x[:m], w, b, out_dtype=torch.float32)

    whole = run(9)
    for m in range(1, 9):
        assert torch.equal(run(m), whole[:m]), m
    want = (x.double() @ w.double().T + b.double() + (start.double() if residual else 0.0)).float()
    assert torch.allclose(whole, want, atol=k * 2.0 ** -24 * float((x.abs() @ w.abs().T).max()), rtol=1e-6)


@pytest.mark.parametrize("m,n,k", [(1, 512, 4096), (3, 4096, 512), (8, 64, 64)])
def test_linear_of_few_rows_reads_a_matrix_written_just_before(m, n, k):
    """The matrix is the result of the launch in front, into the same memory each time."""
    x, w = randn(m, k, seed=330), torch.empty(n, k, device=DEV)
    rows = [randn(n, k, seed=331 + i) for i in range(8)]
    gain = torch.ones(k, device=DEV)
    got = []
    for r in rows:
        ops().rmsnorm(r, gain, 1e-5, torch.float32, out=w)
        got.append(ops().linear(x, w, out_dtype=torch.float32))
    torch.cuda.synchronize()
    for r, g in zip(rows, got):
        ops().rmsnorm(r, gain, 1e-5, torch.float32, out=w)
        torch.cuda.synchronize()
        assert torch.equal(g, ops().linear(x, w, out_dtype=torch.float32))


# ----------------------------------------------------------------------------- what rides in a product's epilogue

def _sums_in_parts(x, parts, seed):
    """Sums of squares of the rows of x, spread over `parts` partial sums (as a producer would leave them)."""
    total = (x.float() * x.float()).sum(dim=-1)
    weights = torch.rand(x.shape[0], parts, generator=torch.Generator().manual_seed(seed)).to(DEV) + 0.1
    sums = torch.full((x.shape[0], ops().SUMSQ_LD), 1e30, device=DEV)      # unused parts must not be read
    sums[:, :parts] = total[:, None] * weights / weights.sum(dim=-1, keepdim=True)
    return sums


def _emit(m, n):
    return ops().Emit(torch.zeros(m, n, dtype=torch.bfloat16, device=DEV), torch.zeros(m, ops().SUMSQ_LD, device=DEV))


@pytest.mark.parametrize("m,n,k,parts", [(8, 6144, 4096, 32), (1, 256, 64, 1), (16, 384, 512, 3),
                                         (40, 320, 1024, 5), (128, 512, 256, 64), (300, 512, 256, 2),
                                         (2048, 1024, 256, 16), (700, 200, 72, 1)])
@pytest.mark.parametrize("bias", [False, True])
def test_linear_with_a_folded_norm(m, n, k, parts, bias):
    """The norm folded into the product: un-normalised bfloat16 rows, the gain in the weights, the rows
    of the result scaled by 1 / sqrt(mean square + eps) in the epilogue (every kernel shape: decode
    tiles summed by the last block or by the sum kernel, one split, tokens on the 128-row side, pairs
    of SMs), against normalising first with the plain norm."""
    x = randn(m, k, seed=140, scale=3.0)
    x[m // 2] *= 1e-3
    gain = 1.0 + randn(k, seed=141, scale=0.2)
    w = randn(n, k, dtype=torch.bfloat16, seed=142, scale=0.1)
    b = randn(n, seed=143) if bias else None
    eps = 1e-5
    folded = (w.float() * gain[None, :]).to(torch.bfloat16)
    norm = ops().FoldedNorm(x.to(torch.bfloat16), _sums_in_parts(x, parts, 144), parts, eps, k)
    got = ops().linear(norm.rows, folded, b, norm=norm)
    want = plain_ops.rmsnorm(x, gain, eps, torch.float32) @ w.float().T + (b if bias else 0.0)
    assert torch.allclose(got.float(), want, atol=3e-2 * float(want.abs().max()), rtol=3e-2)
    assert torch.allclose(plain_ops.linear(norm.rows, folded, b, norm=norm).float(), want,
                          atol=3e-2 * float(want.abs().max()), rtol=3e-2)
    assert ops().tensor_core_status() == 0


@pytest.mark.parametrize("m,f,k", [(8, 14336, 4096), (40, 320, 1024), (300, 1024, 520), (2048, 1024, 256)])
def test_gated_epilogue_with_a_folded_norm(m, f, k):
    x = randn(m, k, seed=150, scale=2.0)
    gain = 1.0 + randn(k, seed=151, scale=0.2)
    gate = randn(f, k, dtype=torch.bfloat16, seed=152, scale=0.05)
    up = randn(f, k, dtype=torch.bfloat16, seed=153, scale=0.05)
    mixed = torch.stack([gate.view(-1, 16, k), up.view(-1, 16, k)], dim=1).reshape(2 * f, k)
    folded = (mixed.float() * gain[None, :]).to(torch.bfloat16).contiguous()
    norm = ops().FoldedNorm(x.to(torch.bfloat16), _sums_in_parts(x, 7, 154), 7, 1e-6, k)
    got = ops().linear(norm.rows, folded, glu=True, norm=norm)
    h = plain_ops.rmsnorm(x, gain, 1e-6, torch.float32)
    g, u = h @ gate.float().T, h @ up.float().T
    want = g / (1 + torch.exp(-g)) * u
    assert torch.allclose(got.float(), want, atol=3e-2 * float(want.abs().max()), rtol=3e-2)


@pytest.mark.parametrize("m,n,k", [(8, 4096, 4096), (1, 4096, 14336), (16, 384, 512), (8, 200, 256),
                                   (40, 4096, 1024), (64, 520, 256), (300, 512, 256), (5, 64, 64)])
def test_linear_leaves_the_next_norms_input(m, n, k):
    """A product that adds into the residual also leaves the updated rows as bfloat16 and the sums of
    their squares in parts (by the tile's last block, by the sum kernel, or by a kernel behind the
    product where the shape's kernel has no such epilogue): twice in a row on the same buffers."""
    a = randn(m, k, dtype=torch.bfloat16, seed=160)
    w = randn(n, k, dtype=torch.bfloat16, seed=161, scale=0.1)
    b = randn(n, seed=162)
    residual = randn(m, n, seed=163, scale=2.0)
    want = residual.clone()
    emit = ops().Emit(torch.zeros(m, n, dtype=torch.bfloat16, device=DEV),
                      torch.full((m, ops().SUMSQ_LD), float("nan"), device=DEV))
    for _ in range(2):
        want = want + (a.float() @ w.float().T + b)
        ops().linear(a, w, b, residual=residual, emit=emit)
        scale = float(want.abs().max())
        assert torch.allclose(residual, want, atol=2e-2 * scale, rtol=2e-2)
        assert 1 <= emit.parts <= ops().SUMSQ_LD
        assert torch.equal(emit.rows, residual.to(torch.bfloat16))
        sums = emit.sumsq[:, :emit.parts].sum(dim=-1)
        assert torch.allclose(sums, (residual * residual).sum(dim=-1), rtol=1e-4)
    assert ops().tensor_core_status() == 0


@pytest.mark.parametrize("tokens", [1, 8, 16, 40, 128, 300, 1100])
@pytest.mark.parametrize("heads,kv_heads,dim,interleaved,bias", [(8, 2, 128, False, False), (4, 4, 64, False, True),
                                                                 (6, 2, 32, True, True), (3, 1, 128, True, False),
                                                                 (6, 2, 48, False, False)])
def test_qkv_product_rotates_and_writes_the_cache(tokens, heads, kv_heads, dim, interleaved, bias):
    """The q/k/v product with the rotation and the cache write in its epilogue (and a folded norm
    with it) against the product followed by the plain rope_cache_write: sequences at different
    positions and pages, head sizes that fit a tile and one that does not (48: a kernel of its own
    runs behind the product). 1,100 tokens run on pairs of SMs, as 256 x 256 tiles or with the weights on
    the row side, which leave the rotation to the kernel behind them."""
    k = 256
    width = (heads + 2 * kv_heads) * dim
    counts = [tokens] if tokens < 3 else [tokens - 2, 1, 1]
    starts = [130, 63, 0][:len(counts)]
    lens = [s + c for s, c in zip(starts, counts)]
    table, pages_wide, k_cache, v_cache = make_cache(len(counts), lens, kv_heads, dim, torch.bfloat16, 170)
    tok_pos = torch.tensor([p for s, c in zip(starts, counts) for p in range(s, s + c)], dtype=torch.int32, device=DEV)
    tok_seq = torch.tensor([i for i, c in enumerate(counts) for _ in range(c)], dtype=torch.int32, device=DEV)
    x = randn(tokens, k, seed=171, scale=2.0)
    gain = 1.0 + randn(k, seed=172, scale=0.2)
    w = randn(width, k, dtype=torch.bfloat16, seed=173, scale=0.1)
    b = randn(width, seed=174) if bias else None
    folded = (w.float() * gain[None, :]).to(torch.bfloat16)
    norm = ops().FoldedNorm(x.to(torch.bfloat16), _sums_in_parts(x, 4, 175), 4, 1e-5, k)
    angle = torch.arange(max(lens) + 1, dtype=torch.float64)[:, None] * (
        10000.0 ** (-2.0 * torch.arange(dim // 2, dtype=torch.float64) / dim))[None, :]
    rope = torch.cat([angle.cos(), angle.sin()], 1).float().to(DEV)
    # plain: normalise, project, round as the unfused path does, rotate, write
    want_qkv = (plain_ops.rmsnorm(x, gain, 1e-5, torch.float32) @ w.float().T + (b if bias else 0.0)).to(torch.bfloat16)
    want_k, want_v = k_cache.clone(), v_cache.clone()
    plain_ops.rope_cache_write(want_qkv, rope, tok_pos, tok_seq, table, pages_wide, want_k, want_v, heads,
                               kv_heads, dim, interleaved)
    for write in (True, False):
        got_k, got_v = k_cache.clone(), v_cache.clone()
        got = ops().linear(norm.rows, folded, b, norm=norm, rope=ops().RopeWrite(
            rope, tok_pos, tok_seq, table, pages_wide, got_k, got_v, heads, kv_heads, dim, interleaved, write))
        q = heads * dim
        scale = float(want_qkv.float().abs().max())
        assert torch.allclose(got[:, :q].float(), want_qkv[:, :q].float(), atol=3e-2 * scale, rtol=3e-2)
        if write:
            assert torch.allclose(got_k.float(), want_k.float(), atol=3e-2 * scale, rtol=3e-2)    # other rows keep 7.0
            assert torch.allclose(got_v.float(), want_v.float(), atol=3e-2 * scale, rtol=3e-2)
        else:
            assert torch.equal(got_k, k_cache) and torch.equal(got_v, v_cache)
    assert ops().tensor_core_status() == 0


def test_cast_sumsq_and_embedding_leave_the_first_norms_input():
    x = randn(9, 1000, seed=180, scale=3.0)
    emit = ops().Emit(torch.empty(9, 1000, dtype=torch.bfloat16, device=DEV), torch.zeros(9, ops().SUMSQ_LD, device=DEV))
    ops().cast_sumsq(x, emit)
    assert emit.parts == 1 and torch.equal(emit.rows, x.to(torch.bfloat16))
    assert torch.allclose(emit.sumsq[:, 0], (x * x).sum(dim=-1), rtol=1e-5)
    table = randn(301, 72, dtype=torch.bfloat16, seed=181)
    tokens = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32, device=DEV)
    emit = ops().Emit(torch.empty(5, 72, dtype=torch.bfloat16, device=DEV), torch.zeros(5, ops().SUMSQ_LD, device=DEV))
    got = ops().embed(tokens, table, scale=2.0, emit=emit)
    want = plain_ops.embed(tokens, table, scale=2.0)
    assert torch.equal(got, want) and torch.equal(emit.rows, want.to(torch.bfloat16))
    assert torch.allclose(emit.sumsq[:, 0], (want * want).sum(dim=-1), rtol=1e-5)
