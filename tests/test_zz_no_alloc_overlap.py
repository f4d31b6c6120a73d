"""kw_kspace_gradient_noalloc launches its second and third kernels with
programmatic stream serialization: calls enqueued one after the other, with
the caller's own kernels between them, must give the bits of calls that are
waited for one by one.  (A call cannot be recorded into a graph: asking for
the stream's device is not permitted while it captures.)"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(384, 320), (45, 60), (1024, 768), (16, 2)])
def test_calls_in_a_row_give_the_bits_of_single_ones(n):
    import torch
    from kwave import _lib

    nx, ny = n
    g = torch.Generator(device="cuda").manual_seed(nx)
    fields = [torch.randn((ny, nx), generator=g, device="cuda") for _ in range(8)]
    f = torch.empty((ny, nx), device="cuda")

    def run(wait):
        res = []
        gx, gy = torch.empty_like(f), torch.empty_like(f)
        for x in fields:
            f.copy_(x)
            gx.fill_(float("nan"))
            gy.fill_(float("nan"))
            _lib.kspace_gradient_noalloc(f.data_ptr(), gx.data_ptr(), gy.data_ptr(), nx, ny, 1e-4, 1e-4, 1500.0, 2e-8,
                                         torch.cuda.current_stream().cuda_stream)
            res.append((gx.clone(), gy.clone()))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return res

    for a, b in zip(run(True), run(False)):
        assert torch.isfinite(a[0]).all() and torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
