"""Column passes launched as programmatic dependents up to a size of the waves and
plainly above it, and 256^2 tiles dealt differently past 65536 of them: each wave of a
batch on either side of a line equals its own run."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(256, 2047), (256, 2048), (384, 17), (384, 18), (768, 71), (768, 72), (1024, 40), (1024, 41)])
def test_batches_on_both_sides_of_the_overlap_limit(n, batch):
    from multislice_gb300 import Context

    g = torch.Generator(device="cuda").manual_seed(n + batch)
    trans = torch.exp(0.2j * torch.randn(2, n, n, generator=g, device="cuda")).to(torch.complex64)
    psi = torch.exp(0.1j * torch.randn(batch, n, n, generator=g, device="cuda")).to(torch.complex64)
    seq = np.array([0, 1, 1, 0], np.int32)
    ctx = Context(0)
    many = psi.clone()
    ctx.multislice(trans, 2.0, seq, 20.0, 20.0, 200.0, psi=many)
    for b in (0, batch // 2, batch - 1):
        one = psi[b : b + 1].clone()
        ctx.multislice(trans, 2.0, seq, 20.0, 20.0, 200.0, psi=one)
        torch.cuda.synchronize()
        assert torch.equal(many[b : b + 1], one)
