"""The closure on batches beyond one launch dimension's 65535 blocks."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _waves(b, h, w, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.randn((b, h, w), dtype=torch.complex64, device="cuda", generator=g)
    torch.cuda.synchronize()
    return z


def test_more_images_than_a_grid_dimension(ctx):
    from multislice_gb300.api import Closure
    net = Closure(ctx, seed=3)
    b = 65540
    psi = _waves(b, 3, 128, 1)
    some = [0, 1, 65534, 65535, 65536, b - 1]
    want = psi[some].clone()
    torch.cuda.synchronize()
    net.apply(want)
    net.apply(psi)
    assert torch.equal(psi[some], want)
    assert torch.isfinite(torch.view_as_real(psi)).all()
    net.close()
