"""Columns launched as dependents or plainly by the size of the waves and, two-stage ones
of 384 and 768, by how full their last round of tiles is; 256^2 tiles dealt differently
past 65536: a wave of a batch on either side of each line (of a GPU of 152 SMs) equals
its own run, all inputs made before the calls."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(384, 18), (384, 19), (384, 56), (384, 57), (384, 60), (384, 61), (384, 123),
                                     (384, 124), (768, 4), (768, 5), (768, 9), (768, 10), (768, 11), (768, 12), (768, 71), (768, 72), (256, 2047),
                                     (256, 2048), (1024, 40), (1024, 41)])
def test_batches_on_both_sides_of_the_rounds(n, batch):
    _check(n, n, batch)


@pytest.mark.parametrize("nx,ny,batch", [(384, 128, 53), (384, 128, 54), (384, 2048, 3), (384, 2048, 4), (768, 128, 36)])
def test_rectangles(nx, ny, batch):
    _check(nx, ny, batch)


def _check(n, ny, batch):
    from multislice_gb300 import Context
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    trans = torch.exp(0.2j * torch.randn(2, n, ny, generator=g, device="cuda")).to(torch.complex64)
    many = torch.exp(0.1j * torch.randn(batch, n, ny, generator=g, device="cuda")).to(torch.complex64)
    some = [0, batch // 2, batch - 1]
    ones = [many[b : b + 1].clone() for b in some]
    seq = np.array([0, 1, 1, 0], np.int32)
    torch.cuda.synchronize()
    with Context(0) as c:
        c.multislice(trans, 2.0, seq, 20.0, 20.0, 200.0, psi=many)
        for b, one in zip(some, ones):
            c.multislice(trans, 2.0, seq, 20.0, 20.0, 200.0, psi=one)
            assert torch.equal(many[b : b + 1], one)
