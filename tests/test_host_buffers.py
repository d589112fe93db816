"""Host arrays around the sizes where their transfers change form (direct, one staging slot, all slots,
several rounds of them): the bytes and values of the same call on device memory, from pageable and
pinned arrays; and an output large enough for the copy on the worker threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOT = 8 << 20
PLAN = ",".join(["cubic2_012"] * 4)


@pytest.mark.parametrize("nbytes", [(4 << 20) - 4096, 4 << 20, SLOT, SLOT + 4096, 3 * SLOT, 3 * SLOT + 4096, 5 * SLOT - 4096])
def test_staged_transfers(gpu_ctx, nbytes):
    import torch

    import asz_b200.api as api
    shape = (nbytes // 4096, 16, 64)
    g = torch.Generator(device="cuda").manual_seed(nbytes)
    x = torch.randn(shape, generator=g, device="cuda").cumsum(2)
    torch.cuda.synchronize()
    p = api.default_params(block_pivot_ratio=3)
    want, _ = gpu_ctx.compress(x, 1e-2, PLAN, "cubic", p)
    host = x.cpu()
    for a in (host.numpy(), host.pin_memory().numpy()):
        assert gpu_ctx.compress(a, 1e-2, PLAN, "cubic", p)[0] == want
    y = torch.empty_like(x)
    gpu_ctx.decompress(want, shape, 1e-2, p, out=y)
    for blob in (want, bytearray(want), memoryview(want)):
        got, _ = gpu_ctx.decompress(blob, shape, 1e-2, p)
        assert np.array_equal(got.view(np.uint32), y.cpu().numpy().view(np.uint32))


def test_large_output(gpu_ctx):
    import torch

    import asz_b200.api as api
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand((256, 256, 320), generator=g, device="cuda")
    torch.cuda.synchronize()
    p = api.default_params(block_pivot_ratio=3)
    a, _ = gpu_ctx.compress(x, 1e-5, PLAN, "cubic", p)
    assert len(a) > 32 << 20
    b, _ = gpu_ctx.compress(x, 1e-5, PLAN, "cubic", p)
    assert a == b
    y = torch.empty_like(x)
    gpu_ctx.decompress(a, x.shape, 1e-5, p, out=y)
    assert np.array_equal(gpu_ctx.debug_recon().view(np.uint32), y.cpu().numpy().ravel().view(np.uint32))
