"""The potential gather where its paths meet: pixels on an atom, at the inner edge of
the radial tables (0.15 A, below it the analytic form) and just inside the cutoff;
cutoffs barely wider than the analytic core; more species than the tables take; grids
narrower than a tile and ragged ones -- against the FP64 oracle."""
import numpy as np
import pytest

from multislice_gb300 import specimen as S
from oracle import msl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,radius,nz", [(64, 64, 0.31, 1), (64, 384, 4.9, 3), (384, 128, 2.5, 8),
                                             (128, 64, 3.0, 9), (2048, 64, 4.0, 2)])
def test_potential_paths_match_oracle(ctx, fparams, nx, ny, radius, nz):
    rng = np.random.default_rng(nx + ny + nz)
    ax, by, cz, ns = 10.0, 12.0, 6.0, 3
    zs = np.array([14, 8, 79, 22, 38, 6, 29, 1, 92])[:nz]
    n = 40
    x, y, z = rng.uniform(-1, ax + 1, n), rng.uniform(-1, by + 1, n), rng.uniform(-0.5, cz + 0.5, n)
    dx, dy = ax / nx, by / ny
    x[0], y[0], z[0] = 3 * dx, 5 * dy, 1.0            # on a pixel
    x[1], y[1], z[1] = 9 * dx - 0.15, 7 * dy, 3.0     # a pixel at the tables' inner edge
    x[2], y[2], z[2] = 11 * dx - radius * 0.9999, 9 * dy, 5.0  # a pixel just inside the cutoff
    spec = S.Specimen(x, y, z, zs[np.arange(n) % nz].astype(np.int32), ax, by, cz)
    v = ctx.potential(spec, nx, ny, ns, radius)
    ref = O.potential(x, y, z, spec.Z, fparams, ax, by, cz, nx, ny, ns, radius)
    assert v.shape == ref.shape and np.isfinite(v).all()
    assert O.rel_l2(v, ref) < 1e-5


# rows that form the transmission function themselves (256, 512, 1024) and those that
# start from the elementwise kernel; many turns of phase, both signs; a potential that
# bulk copies cannot take
@pytest.mark.parametrize("nx,ny,shift", [(64, 128, 0), (64, 256, 0), (128, 512, 0), (64, 1024, 0), (64, 384, 0),
                                         (64, 256, 1), (64, 2048, 0)])
def test_transmission_paths_match_oracle(ctx, nx, ny, shift):
    import torch
    rng = np.random.default_rng(nx + ny)
    ax, by, kev = 9.0, 11.0, 200.0
    v = rng.uniform(-40000.0, 40000.0, (2, nx, ny)).astype(np.float32)
    flat = torch.empty(v.size + 4, dtype=torch.float32, device="cuda")
    dev = flat[shift:shift + v.size].view(2, nx, ny)
    dev.copy_(torch.from_numpy(v))
    torch.cuda.synchronize()
    t = ctx.transmission(dev, ax, by, kev)
    ref = O.transmission(v.astype(np.float64), kev, ax, by, np.complex128)
    assert O.rel_l2(t, ref) < 1e-5
