"""The potential gather at the ends of its number range: atoms a denormal squared
distance from a pixel -- against the FP64 oracle."""
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
