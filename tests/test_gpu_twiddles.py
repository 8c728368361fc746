"""The twiddle tables of the two-stage 384 and 768 transforms: phases of transformed
unit impulses, averaged over random amplitudes so that only what is the same in every
transform (the tables and constants) is left."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [384, 768])
@pytest.mark.parametrize("rows", [True, False])
@pytest.mark.parametrize("direction", [1, -1])
def test_table_phases(n, rows, direction):
    """A phase is a table entry's, rounded to float (2^-25 / sqrt 3 rms), that of the radix
    3, 8, 16 and 32 butterflies' constants (as much again), and what the average over 256
    amplitudes leaves of the rounding of the transforms (3 * 2^-24 rms a value, / 16)."""
    from multislice_gb300 import Context
    m, pos = 256, [23, 24, 47, n // 2 + 1, n - 1, n - 23]
    g = torch.Generator(device="cuda").manual_seed(n)
    amp = torch.exp(2j * np.pi * torch.rand(m, generator=g, device="cuda", dtype=torch.float64)).to(torch.complex64)
    amp *= 1 + torch.rand(m, generator=g, device="cuda")
    square = 0.0
    with Context(0) as c:
        for j in pos:
            psi = torch.zeros((m, 64, n) if rows else (m, n, 64), dtype=torch.complex64, device="cuda")
            (psi[:, 0] if rows else psi[:, :, 0])[:, j] = amp
            torch.cuda.synchronize()
            c.fft2d(psi, 10.0, 10.0, direction)
            line = (psi[:, 0] if rows else psi[:, :, 0]).to(torch.complex128)  # every other row or column is equal
            k = torch.arange(n, device="cuda", dtype=torch.float64)
            want = torch.exp(direction * 2j * np.pi * ((k * j) % n) / n)
            mean = (line / amp.to(torch.complex128)[:, None] * want.conj()).mean(0)
            square += torch.angle(mean).pow(2).mean().item() / len(pos)
    assert square ** 0.5 < 2.0 ** -24 * (2 * 0.25 / 3 + (3 / 16) ** 2) ** 0.5
