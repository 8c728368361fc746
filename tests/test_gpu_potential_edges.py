"""The potential gather at the ends of its number range: atoms a denormal squared
distance from a pixel, and cells so large that float positions are coarse against the
culling's margin -- against the FP64 oracle."""
import numpy as np
import pytest

from multislice_gb300 import specimen as S
from oracle import msl_oracle as O

pytestmark = pytest.mark.gpu

# distances whose square is a float denormal (below 1.08e-19 A), zero or just normal
HAIRS = [(1e-20, 0.0), (0.0, 2e-20), (5e-21, 7e-21), (1e-19, 0.0), (3.8e-23, 0.0), (0.0, 1e-22), (1e-30, 1e-30),
         (1.2e-19, 0.0), (0.0, 0.0)]


@pytest.mark.parametrize("extra", [1, 8])  # one species (tabulated profiles), nine (analytic kernel)
def test_atoms_a_hair_from_a_pixel(ctx, fparams, extra):
    ax, by, ns, n, radius = 10.0, 12.0, len(HAIRS), 64, 3.0
    x, y = np.array(HAIRS).T
    z = np.arange(ns) + 0.5
    Z = np.full(ns, 14, np.int32)
    if extra == 8:  # eight more species away from the corner, in the first slice
        x, y, z = np.append(x, np.linspace(2, 8, 8)), np.append(y, np.linspace(3, 9, 8)), np.append(z, np.full(8, 0.5))
        Z = np.append(Z, np.array([8, 79, 22, 38, 6, 29, 1, 92], np.int32)).astype(np.int32)
    v = ctx.potential(S.Specimen(x, y, z, Z, ax, by, float(ns)), n, n, ns, radius)
    ref = O.potential(x, y, z, Z, fparams, ax, by, float(ns), n, n, ns, radius)
    assert np.isfinite(v).all()
    assert O.rel_l2(v, ref) < 1e-5


@pytest.mark.parametrize("nx,ny", [(2048, 64), (64, 2048)])
def test_atoms_just_inside_the_cutoff_of_a_tile_in_a_large_cell(ctx, fparams, nx, ny):
    """Each atom reaches one pixel only, the last or first of a 64 x 32-pixel tile, from
    0.1 mA inside the cutoff; at 20 um a float position is off by up to 1 mA."""
    px, radius, ns = 9.77, 1.0, 1
    ax, by = nx * px, ny * px
    dx, dy = ax / nx, by / ny
    t = np.arange(0, 2048, 64 if nx == 2048 else 32)
    near = radius - 1e-4
    along = np.concatenate([(t + (63 if nx == 2048 else 31)) * (dx if nx == 2048 else dy) + near,
                            np.maximum(t * (dx if nx == 2048 else dy) - near, 0.0)[1:]])
    across = (np.arange(len(along)) % 61 + 1) * (dy if nx == 2048 else dx)
    x, y = (along, across) if nx == 2048 else (across, along)
    z = np.full(len(x), 0.5)
    Z = np.full(len(x), 79, np.int32)
    v = ctx.potential(S.Specimen(x, y, z, Z, ax, by, 1.0), nx, ny, ns, radius)
    ref = O.potential(x, y, z, Z, fparams, ax, by, 1.0, nx, ny, ns, radius)
    assert np.count_nonzero(ref) >= len(x)
    assert O.rel_l2(v, ref) < 1e-5


@pytest.mark.parametrize("n,shift", [(512, 0), (513, 0), (511, 1), (512, 1), (1100, 1), (0, 0)])
def test_more_atoms_than_the_output_holds(ctx, fparams, n, shift):
    """Unsorted atoms pass through the output's memory: 512 of them where it is one slice
    of 64^2 on 16 bytes, 511 where it starts 4 bytes on; then the rest."""
    import torch
    rng = np.random.default_rng(n)
    ax, by, radius = 10.0, 12.0, 2.0
    x, y, z = rng.uniform(-1, ax + 1, n), rng.uniform(-1, by + 1, n), rng.uniform(0.0, 1.0, n)
    Z = rng.choice(np.array([8, 22, 38], np.int32), n).astype(np.int32)
    flat = torch.full((64 * 64 + 4,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    v = ctx.potential(S.Specimen(x, y, z, Z, ax, by, 1.0), 64, 64, 1, radius,
                      out=flat[shift:shift + 64 * 64].view(1, 64, 64)).cpu().numpy()
    ref = O.potential(x, y, z, Z, fparams, ax, by, 1.0, 64, 64, 1, radius)
    assert np.abs(v - ref).max() <= 1e-5 * np.abs(ref).max()
    assert torch.isnan(flat[:shift]).all() and torch.isnan(flat[shift + 64 * 64:]).all()
