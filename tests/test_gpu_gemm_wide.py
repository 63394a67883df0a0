"""The tcgen05 GEMM for bf16 weights and f32 activations (projections of more rows than the CUDA-core kernel is for): against
64 bits at the edges of its tiles (128 weight rows, 64 activation rows, 64 columns) and of its cut over the SMs, and, through
models of full width against the oracle, every epilogue that it has (residual add, SwiGLU, rotary embedding and cache write,
planes and sums of squares for the next projection).

Tolerance, per activation row: the activations enter as three bf16 planes whose sum is the f32 value, products are exact, and
single K blocks are summed in f32 by the tensor pipe, so that the error of a result is a few 2^-24 of the 2-norm of its row;
2e-6 of that norm is about 30 times 2^-24."""
import numpy as np
import pytest

from helpers import normal_f32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from paged_infer_b200 import api
    c = api.Context(0)
    yield c
    c.close()


def bf16_matrix(rows, cols, seed):
    from paged_infer_b200.loader import bf16_bits_to_f32, f32_to_bf16_bits
    bits = f32_to_bf16_bits(normal_f32((rows, cols), seed, 0.02))
    return bits, bf16_bits_to_f32(bits)


# one tile; a row more; K that ends inside a block and off the 32-byte grid; fewer tiles than SMs, each shared; more
@pytest.mark.parametrize("rows,cols,M", [(128, 4096, 512), (129, 5608, 449), (2048, 1000, 129), (2047, 2056, 64), (2560, 2048, 65), (11264, 2048, 9),
                                         (24000, 1608, 5), (32000, 2048, 130), (40, 65536, 300)])
def test_bf16_weights(ctx, rows, cols, M):
    from paged_infer_b200 import api
    bits, w = bf16_matrix(rows, cols, rows + M)
    x = normal_f32((M, cols), M, 1.0)
    x[0] *= 1e-6
    x[-1] *= 3e30
    want = x.astype(np.float64) @ w.astype(np.float64).T
    p = api.Projection.f32(ctx, bits)
    before = ctx.kernel_launches()
    got = p.apply_batched(x)
    assert ctx.kernel_launches() - before == 2      # the split and the GEMM: the CUDA-core kernel would be one
    assert np.array_equal(got, p.apply_batched(x))   # a tile's parts are summed in one order
    norm = np.sqrt((want ** 2).mean(axis=1, keepdims=True))
    assert float((np.abs(got - want) / np.maximum(np.abs(want), norm)).max()) < 2e-6
    # As a whole, where sums over blocks that are lost show: a running sum on the tensor pipe is cut by 1.5e-8 of itself every 16
    # columns (2e-6 over 2048), those of single blocks 1.3e-7 at most; f32 sums of the blocks add 2^-25 a block at random.
    rest = slice(1, M - 1)
    bound = 2 * np.hypot(1.3e-7, 2.0 ** -25 * np.sqrt(cols / 64) / 2)
    assert np.linalg.norm((got - want)[rest]) < bound * np.linalg.norm(want[rest])


def test_infinities_and_nan_stay_in_their_rows(ctx):
    from paged_infer_b200 import api
    bits, w = bf16_matrix(4096, 2048, 5)
    w[w == 0] = 1e-3
    from paged_infer_b200.loader import f32_to_bf16_bits
    bits = f32_to_bf16_bits(w)
    x = normal_f32((64, 2048), 6, 1.0)
    x[3, 7], x[5, 9], x[8] = np.inf, np.nan, 0.0
    x[8, 0] = np.finfo(np.float32).max           # rounds up beyond the largest bf16
    got = api.Projection.f32(ctx, bits).apply_batched(x)
    rest = np.ones(64, bool)
    rest[[3, 5]] = False
    assert np.isfinite(got[rest]).all()
    assert np.array_equal(got[3], np.where(w[:, 7] > 0, np.inf, -np.inf).astype(np.float32))
    assert np.isnan(got[5]).all()
    np.testing.assert_allclose(got[8], w[:, 0] * x[8, 0], rtol=1e-6)


@pytest.mark.parametrize("called_before", [False, True])
def test_captured_projection_holds_no_scratch(called_before):
    """A host's graph of a bf16 projection is the one kernel that keeps nothing in the context: the same bits whether or not the
    context has run such calls before, and still after later calls of larger sizes."""
    import torch

    from paged_infer_b200 import api
    M, rows, cols = 64, 2048, 2048                  # eager calls of this size run on the tensor pipe
    bits, _ = bf16_matrix(rows, cols, 7)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = api.Context(0, stream.cuda_stream)
        p = api.Projection.f32(ctx, bits)
        x = torch.zeros(M, cols, device="cuda")
        out, want = torch.empty(M, rows, device="cuda"), torch.empty(M, rows, device="cuda")
        ctx.set_option(1, 0)                        # PI_OPT_TENSOR_GEMM off: the CUDA-core kernel, and its set-up before the capture
        p.apply_device(x, want, M)
        ctx.set_option(1, 1)
        if called_before:
            p.apply_device(x, out, M)
        ctx.synchronize()
        graph = torch.cuda.CUDAGraph()
        before = ctx.kernel_launches()
        with torch.cuda.graph(graph, stream=stream):
            p.apply_device(x, out, M)
        assert ctx.kernel_launches() - before == 1
        larger = api.Projection.f32(ctx, bf16_matrix(2048, 4096, 8)[0])
        for big in (256, 1024):
            larger.apply_device(torch.ones(big, 4096, device="cuda"), torch.empty(big, 2048, device="cuda"), big)
        x.copy_(torch.from_numpy(normal_f32((M, cols), 9, 1.0)))
        graph.replay()
        ctx.set_option(1, 0)
        p.apply_device(x, want, M)
        ctx.synchronize()
        assert torch.equal(out, want)
        del graph
        ctx.close()


@pytest.mark.parametrize("rows,cols,M,portions", [(2048, 1024, 1024, 1), (2048, 1024, 2049, 3), (320, 65536, 700, 2)])
def test_large_batches_pass_in_portions_and_allocate_nothing(rows, cols, M, portions):
    """The planes of a batch have a bounded scratch, laid out when the matrix is created: no call of any size allocates, the first
    one included, and a row's bits are those of the portion it is in."""
    import torch

    from paged_infer_b200 import api
    bits, w = bf16_matrix(rows, cols, rows + M)
    x = torch.from_numpy(normal_f32((M, cols), M, 1.0)).cuda()
    out, part = torch.empty(M, rows, device="cuda"), torch.empty(M, rows, device="cuda")
    want = x.double() @ torch.from_numpy(w).cuda().double().T
    warm = api.Context(0)                               # what the driver sets aside for kernels that run for the first time
    api.Projection.f32(warm, bits).apply_device(x, out, M)
    warm.synchronize()
    ctx = api.Context(0)
    p = api.Projection.f32(ctx, bits)
    torch.cuda.synchronize()
    free, before = torch.cuda.mem_get_info()[0], ctx.kernel_launches()
    p.apply_device(x, out, M)
    ctx.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    assert ctx.kernel_launches() - before == 2 * portions
    assert ((out - want).abs() / want.abs().maximum(want.square().mean(1, keepdim=True).sqrt())).max() < 2e-6
    step = -(-(-(-M // portions)) // 64) * 64 if portions > 1 else M
    for first in range(0, M, step):
        n = min(step, M - first)
        if n * 2 < step:                                # a short rest alone may lie on the other side of the dispatch line
            continue
        p.apply_device(x[first:first + n], part[first:first + n], n)
        ctx.synchronize()
        assert torch.equal(out[first:first + n], part[first:first + n])
    ctx.close()
    warm.close()


def test_int8_graphs_survive_bf16_calls():
    """bf16 projections leave the scratch that int8 ones use alone, also where a host's graph holds it."""
    import torch

    from paged_infer_b200 import api
    M, rows, cols = 64, 2048, 1024
    rng = np.random.default_rng(3)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = api.Context(0, stream.cuda_stream)
        p = api.Projection.int8(ctx, rng.integers(-127, 128, (rows, cols), dtype=np.int8), np.full(rows, 1e-3, np.float32))
        x = torch.from_numpy(normal_f32((M, cols), 1, 1.0)).cuda()
        out, want = torch.empty(M, rows, device="cuda"), torch.empty(M, rows, device="cuda")
        p.apply_device(x, want, M)
        ctx.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            p.apply_device(x, out, M)
        wide = api.Projection.f32(ctx, bf16_matrix(2048, 4096, 8)[0])
        wide.apply_device(torch.ones(256, 4096, device="cuda"), torch.empty(256, 2048, device="cuda"), 256)
        graph.replay()
        ctx.synchronize()
        assert torch.equal(out, want)
        del graph
        ctx.close()


def bf16_llama(ctx, seed, hidden, heads, kv_heads, inter, vocab, layers=1, max_batch=64, rope_style=0, weights="bf16", oracle=None):
    """A model of full width with bf16 projections (or int8 ones) and a bf16 head, random norm weights; its oracle beside it."""
    from paged_infer_b200 import api
    from paged_infer_b200.loader import HostWeights, LlamaConfig, f32_to_bf16_bits
    cfg = LlamaConfig(hidden, layers, heads, kv_heads, inter, vocab, 1e-5, 10000.0)
    cfg.rope_style = rope_style
    kv = kv_heads * (hidden // heads)
    shapes = {"wq": (hidden, hidden), "wk": (kv, hidden), "wv": (kv, hidden), "wo": (hidden, hidden), "w1": (inter, hidden),
              "w2": (hidden, inter), "w3": (inter, hidden)}

    def matrix(shape, i):
        w = normal_f32(shape, seed * 1000 + i, 0.02)
        return f32_to_bf16_bits(w) if weights == "bf16" else oracle.quantize_rows_i8(w, *shape)

    projs = [{k: matrix(s, l * 10 + j) for j, (k, s) in enumerate(shapes.items())} for l in range(layers)]
    norms = [(1.0 + normal_f32((hidden,), seed * 1000 + 900 + i, 0.2)).astype(np.float32) for i in range(2 * layers + 1)]
    head = f32_to_bf16_bits(normal_f32((vocab, hidden), seed * 1000 + 999, 0.02))
    hw = HostWeights(f32_to_bf16_bits(normal_f32((vocab, hidden), seed * 1000 + 998, 0.5)), norms[0], norms[1:layers + 1], norms[layers + 1:], projs, None)
    om = oracle and oracle.Model(cfg.as_dict(), hw.token_embeddings, hw.final_norm, hw.attention_norm, hw.ffn_norm, projs, head)
    return cfg, om, api.LlamaWeights(ctx, cfg, hw, max_batch=max_batch, lm_head=head)


def test_model_chunk_larger_than_a_portion(ctx):
    """A chunk of 1300 rows of a bf16 model: the first layer's [q;k;v] goes through the scratch in two portions, with the rotary
    embedding and the KV write of each; the CUDA-core kernels on the same inputs."""
    from paged_infer_b200 import api
    cfg, _, gm = bf16_llama(ctx, 51, 1024, 16, 4, 2816, 2048, layers=2, max_batch=1300)
    n, block, nblocks = 1300, 16, 90
    rng = np.random.default_rng(2)
    prompt, table = rng.integers(0, cfg.vocab_size, n).astype(np.uint32), [int(b) for b in rng.permutation(nblocks)[:n // block + 1]]
    got = []
    for tensor in (1, 0):
        ctx.set_option(1, tensor)                       # PI_OPT_TENSOR_GEMM
        gkv = api.KvCache(ctx, gm.kv_layout(nblocks, block))
        gkv.upload(np.zeros(gm.kv_layout(nblocks, block).total_floats(), np.float32))
        got.append((gm.prefill_batched(prompt, 0, table, gkv, n), gkv.download()))
    ctx.set_option(1, 1)
    for a, b in zip(*got):                              # five projections in a row, each a few 2^-24 off on either side
        assert np.abs(a - b).max() < 2e-5 * np.sqrt((b.astype(np.float64) ** 2).mean())


def test_infinite_weights(ctx):
    """Weights that are infinite or NaN give what 64 bits and the CUDA-core kernel give, and touch their own columns only."""
    from paged_infer_b200 import api
    bits, w = bf16_matrix(4096, 2048, 11)
    x = normal_f32((70, 2048), 12, 1.0)
    x[9, 100], x[10, 100] = 0.0, np.inf
    x[:, 2047] = np.float32(1.5)                     # exactly one bf16: the other planes are zero
    for row, col, value in [(3, 100, np.inf), (130, 7, -np.inf), (131, 7, np.nan), (4000, 2047, np.inf)]:
        w[row, col] = value
        bits[row, col] = {np.inf: 0x7f80, -np.inf: 0xff80}.get(value, 0x7fc0)
    w[4000, 3], bits[4000, 3] = -np.inf, 0xff80      # two signs in one row: NaN where both act in one direction
    with np.errstate(invalid="ignore"):
        want = x.astype(np.float64) @ w.astype(np.float64).T
    for tensor in (1, 0):                            # PI_OPT_TENSOR_GEMM
        ctx.set_option(1, tensor)
        got = api.Projection.f32(ctx, bits).apply_batched(x)
        ctx.set_option(1, 1)
        finite = np.isfinite(want)
        assert np.array_equal(got[~finite], want[~finite].astype(np.float32), equal_nan=True)
        norm = np.sqrt((np.where(finite, want, 0) ** 2).mean(axis=1, keepdims=True))
        assert (np.abs(got[finite] - want[finite]) / np.maximum(np.abs(want), norm)[finite]).max() < 2e-6


# hidden 2048: heads of 64, whole tiles, rotary embedding in the epilogue; hidden 2000: heads of 80 (rotary embedding behind it),
# no matrix a multiple of the tile; int8 layers under a bf16 head
MODELS = [dict(hidden=2048, heads=32, kv_heads=4, inter=5632, vocab=4096), dict(hidden=2048, heads=16, kv_heads=4, inter=2824, vocab=4100, rope_style=1),
          dict(hidden=2000, heads=25, kv_heads=5, inter=2824, vocab=4100, rope_style=1), dict(hidden=2048, heads=32, kv_heads=4, inter=2816, vocab=8200, weights="int8")]


@pytest.fixture(scope="module", params=range(len(MODELS)))
def bf16_model(request, ctx, oracle):
    return MODELS[request.param], bf16_llama(ctx, 61 + request.param, layers=2, max_batch=130, oracle=oracle, **MODELS[request.param])


def close_to_oracle(got, want, depth=8):
    """Logits (or cache contents) behind `depth` projections in a row: the 2-norm of each one's error is 2e-7 of its result on either
    side and the norms, gates and attention between them pass it on about as it is; values within six of their deviations."""
    scale = np.sqrt((want.astype(np.float64) ** 2).mean())
    return np.abs(got - want).max() < 2 * depth * 2e-7 * 6 * scale


@pytest.mark.parametrize("chunk", [100, 130])
def test_model_prefill(ctx, bf16_model, chunk):
    """A prompt of 230 in chunks that are no multiple of a tile of 64 rows; logits and the cache."""
    from paged_infer_b200 import api
    kind, (cfg, om, gm) = bf16_model
    n, block, nblocks = 230, 16, 18
    rng = np.random.default_rng(4)
    prompt, table = rng.integers(0, cfg.vocab_size, n).astype(np.uint32), [int(b) for b in rng.permutation(nblocks)[:n // block + 1]]
    layout = gm.kv_layout(nblocks, block)
    okv, gkv = np.zeros(layout.total_floats(), np.float32), api.KvCache(ctx, layout)
    gkv.upload(okv)
    want = om.prefill_batched(prompt, 0, table, okv, block, 32)
    ctx.profile_begin()
    got = gm.prefill_batched(prompt, 0, table, gkv, chunk)
    assert ctx.profile_end()["gemm_tc"][1] == 8 * -(-n // chunk)     # every projection but the head of the last row
    assert close_to_oracle(got, want)
    assert close_to_oracle(gkv.download()[okv != 0], okv[okv != 0])


@pytest.mark.parametrize("batch", [8, 12, 24, 64])
def test_model_decode(ctx, oracle, bf16_model, batch):
    """Batches on both sides of the dispatch line and across it (some projections of a layer on each kernel): a step with logits, then
    greedy steps, the later ones out of a captured graph."""
    from paged_infer_b200 import api
    kind, (cfg, om, gm) = bf16_model
    block, nblocks, steps = 16, 3 * batch, 6
    rng = np.random.default_rng(5)
    layout = gm.kv_layout(nblocks, block)
    okv = (rng.standard_normal(layout.total_floats()) * 0.5).astype(np.float32)
    before, gkv = okv.copy(), api.KvCache(ctx, layout)
    gkv.upload(okv)
    tables = [[int(x) for x in row] for row in rng.permutation(nblocks).reshape(batch, 3)]
    tokens, pos = [int(t) for t in rng.integers(0, cfg.vocab_size, batch)], [int(p) for p in rng.integers(0, 40, batch)]
    want = om.decode_batch(tokens, pos, tables, okv, block)
    ctx.profile_begin()
    got = gm.decode_batch_into(tokens, pos, tables, gkv, want_logits=True)
    tensor = ctx.profile_end()["gemm_tc"][1]
    assert tensor == 9 if batch == 64 or (kind.get("weights") == "int8" and batch >= 12) else tensor < 9
    assert close_to_oracle(got, want)
    ids = gm.decode_multi(tokens, pos, tables, gkv, steps)
    for i in range(steps):
        want = om.decode_batch(tokens, [p + i for p in pos], tables, okv, block)
        tokens = [oracle.argmax(r) for r in want]
        assert ids[i].tolist() == tokens
    wrote, after = okv != before, gkv.download()
    assert np.array_equal(after[~wrote], okv[~wrote])
    assert close_to_oracle(after[wrote], okv[wrote])    # against the size of what was written, not of the rest of the cache
