"""The wide column transform (row-major output, lengths from 1024 up): sizes on both
sides of the rule that takes it and a last CTA that is not full, against the float64 DFT,
with the per-transform bound of the other FFT tests (5e-7 relative L2)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,batch", [
    (1024, 16, 80), (1024, 16, 1), (1024, 1024, 2), (1536, 24, 53), (1536, 24, 2), (2048, 48, 26), (2048, 48, 25),
    (3072, 16, 38), (3072, 96, 7), (4096, 24, 26), (4096, 32, 1)])
def test_wide_columns_match_float64(cdx, torch_cuda, rows, cols, batch):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(batch, rows, cols, dtype=torch.complex64, device="cuda", generator=g)
    y = torch.full_like(x, float("nan"))
    st = torch.cuda.current_stream().cuda_stream
    for inverse in (False, True):
        cdx.fft2(x, y, inverse=inverse, stream=st)
        w = x.to(torch.complex128)
        ref = torch.fft.ifft2(w, norm="forward") if inverse else torch.fft.fft2(w)
        assert float((y - ref).norm() / ref.norm()) < 5e-7


@pytest.mark.parametrize("rows,cols", [(1024, 1536), (2048, 1536), (2048, 2048)])
def test_final_psi_from_tiles(cdx, torch_cuda, rows, cols):
    """A run's closing transform reads the iteration's narrow tiles: Psi equals the transform of the object."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(7)
    inten = [torch.rand(rows, cols, device="cuda", generator=g)]
    inten.append(inten[0] * 2)
    torch.cuda.synchronize()   # the context reads them on a stream of its own
    with cdx.Context(cdx.default_params(rows, cols, batch=2, beta=0.9)) as ctx:
        for k in range(2):
            ctx.set_pattern(k, inten[k])
        ctx.random_start(3)
        ctx.run("2*ER")
        for k in range(2):
            rho = torch.from_numpy(ctx.get_object(k)).cuda().to(torch.complex128) / (rows * cols) ** 0.5
            psi = torch.from_numpy(ctx.get_fourier(k)).cuda()
            ref = torch.fft.fft2(rho)
            assert float((psi - ref).norm() / ref.norm()) < 5e-7


@pytest.mark.parametrize("rows,cols,batch", [(1024, 1024, 3), (1024, 16, 129), (1024, 24, 90), (1024, 2048, 2)])
def test_wide_columns_of_1024_match_float64(cdx, torch_cuda, rows, cols, batch):
    """From 2^21 pixels on, below which lengths of 1024 take the geometry for small work: row-major input."""
    assert rows * cols * batch > 1 << 21 and (cols + 7) // 8 * batch >= 152
    test_wide_columns_match_float64(cdx, torch_cuda, rows, cols, batch)
