"""Propagator and defocus tables whose descriptions travel as kernel arguments, at the
counts where a launch carries more of them or another launch begins."""
import numpy as np
import pytest

from oracle import msl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [16, 17, 512, 513, 1030])
def test_the_last_layers_of_many(ctx, layers):
    n, rng = 64, np.random.default_rng(layers)
    dz = rng.uniform(0.5, 3.0, layers)
    t = np.exp(0.2j * rng.standard_normal((3, n, n))).astype(np.complex64)
    some = np.array([0, layers // 2, layers - 1])
    trans = np.ones((layers, n, n), np.complex64)
    trans[some] = t
    many = ctx.multislice(trans, dz, some, 8.0, 9.0, 200.0)
    few = ctx.multislice(t, dz[some], [0, 1, 2], 8.0, 9.0, 200.0)
    assert np.array_equal(many, few)


@pytest.mark.parametrize("ndf", [15, 17, 255, 257, 513])
def test_many_defocus_values_vs_oracle(ctx, ndf):
    n, rng = 64, np.random.default_rng(ndf)
    ax, by, kev, step = 8.0, 9.0, 200.0, 4.0
    spread = step * (ndf // 2) / 2.5 * (1 + 1e-9)
    V = np.zeros((1, n, n))
    V[0, rng.integers(0, n, 12), rng.integers(0, n, 12)] = rng.uniform(50, 400, 12)
    t = O.transmission(V, kev, ax, by, np.complex64)
    img, _, _ = ctx.ctem_image(t, 1.5, [0], ax, by, kev, 1.2e7, -600.0, 1.5, df_spread=spread, df_step=step)
    props = [O.propagator_tables(n, n, ax, by, kev, 1.5, precision="f64")]
    w0, _ = O.multislice(np.ones((n, n), np.complex128), t.astype(np.complex128), props, [0], O.band_mask(n, n, ax, by))
    assert O.rel_l2(img, O.ctem_image(w0, ax, by, kev, 1.2e7, -600.0, 1.5, spread, step)) < 2e-5
