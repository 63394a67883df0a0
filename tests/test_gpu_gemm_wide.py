"""The tcgen05 GEMM for bf16 weights and f32 activations (projections of more rows than the CUDA-core kernel is for): against
64 bits at the edges of its tiles (128 weight rows, 64 activation rows, 64 columns) and of its cut over the SMs.

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
