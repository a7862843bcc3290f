"""The warm-start network on streams that a context may be given: its own, the per-thread
default stream and the legacy default stream (which cannot be captured).  One pass is the
same arithmetic everywhere: the output has the same bits, the loss and the gradients
(summed with FP32 atomics) agree within 1e-4 of the largest gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LEGACY, PER_THREAD = 1, 2  # cudaStreamLegacy, cudaStreamPerThread


@pytest.mark.parametrize("stream", [PER_THREAD, LEGACY])
@pytest.mark.parametrize("nx,ny", [(64, 40), (256, 192)])
def test_passes_on_default_streams(lib, nx, ny, stream):
    from iskra_gb300.device import Context
    rng = np.random.default_rng(nx)
    img = rng.normal(size=(ny, nx)).astype(np.float32)
    tgt = rng.normal(size=(ny, nx)).astype(np.float32)
    out = []
    for st in (0, stream):
        ctx = Context(nx, ny, 1e-3, 1e-3, stream=st)
        ctx.lws_create(2, seed=3)
        passes = [(ctx.lws_forward(img), *ctx.lws_loss_grad(img, tgt)) for _ in range(2)]
        out.append(passes)
        ctx.close()
    for own, other in zip(*out):
        assert np.array_equal(own[0], other[0])
        assert abs(own[1] - other[1]) <= 1e-9 * abs(own[1])
        assert np.max(np.abs(own[2] - other[2])) <= 1e-4 * np.max(np.abs(own[2]))
