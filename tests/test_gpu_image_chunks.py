"""Images added onto one accumulator in chunks of 512 MB, the second of which starts
between two defocus values of one wave: the same sums, bit for bit, as one image at a
time (a context with a memory cap), for every row kernel that sums images."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,waves,steps,family", [(64, 10, 1000, 0), (64, 10, 1000, 2), (128, 5, 440, 0), (256, 6, 100, 0),
                                                  (256, 6, 100, 1), (384, 5, 50, 0), (512, 6, 25, 0), (768, 6, 10, 0),
                                                  (1024, 6, 6, 0), (2048, 3, 4, 0)])
def test_chunks_do_not_change_the_sums(n, waves, steps, family):
    from multislice_gb300 import Context
    ndf = 2 * steps + 1  # defocus values
    assert waves * ndf * n * n * 8 > 512 << 20
    g = torch.Generator(device="cuda").manual_seed(n)
    trans = torch.exp(0.2j * torch.randn(1, n, n, generator=g, device="cuda")).to(torch.complex64)
    psi = torch.exp(0.1j * torch.randn(waves, n, n, generator=g, device="cuda")).to(torch.complex64)
    torch.cuda.synchronize()

    def run(cap):
        with Context(0) as c:
            c.set_memory_limit(cap)
            c.set_schedule(n, family, family)
            try:
                p = psi.clone()
                torch.cuda.synchronize()
                exi = np.zeros((n, n))
                img, w, _ = c.ctem_image(trans, 1.5, [0], 0.1 * n, 0.1 * n, 200.0, 1.2e7, -600.0, 1.5, psi=p,
                                         df_spread=4.0 * steps, df_step=10.0, weight=0.7, exit_intensity=exi)
                return img, exi, p.cpu().numpy()
            finally:
                c.set_schedule(n, 0, 0)

    for a, b in zip(run(0), run(1 << 36)):
        assert np.isfinite(a).all() and np.array_equal(a, b)
