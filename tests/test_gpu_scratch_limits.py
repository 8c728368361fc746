"""Work buffers under a cap (msl_set_memory_limit): the least cap each kind of call
has always run in, and what an uncapped call leaves behind."""
import numpy as np
import pytest

from multislice_gb300 import specimen as S

pytestmark = pytest.mark.gpu


def _t(nt, nx, ny=None):
    rng = np.random.default_rng(nx + nt)
    return np.exp(0.2j * rng.standard_normal((nt, nx, ny or nx))).astype(np.complex64)


def _multislice(c):
    return c.multislice(_t(3, 64, 128), [1.5, 1.6, 1.7], [0, 1, 2, 0], 6.0, 12.0, 200.0)


def _thick(c):  # many layers: the propagator tables are most of the scratch
    return c.multislice(_t(200, 64), np.linspace(1, 2, 200), np.arange(200), 6.0, 6.0, 200.0)


def _image(c):
    return c.ctem_image(_t(1, 64), 1.5, [0], 6.0, 6.0, 200.0, 1.2e7, -600.0, 1.5, batch=3, df_spread=40.0, df_step=20.0)[0]


def _partial(c):
    return c.partial_coherence(_t(1, 64), 1.5, [0], 20.0, 20.0, 200.0, 1.2e7, -600.0, 1.5, 0.0, 2.4e-3, df_spread=40.0,
                               df_step=20.0)[0]


def _potential(c):
    return c.potential(S.srtio3(6, 6, 4), 64, 64, 2, 3.0)


def _species(c):  # more species than the radial tables take
    s = S.srtio3(4, 4, 4)
    s.Z = (np.arange(len(s.Z)) % 12 + 6).astype(np.int32)
    return c.potential(s, 64, 64, 8, 3.0)


def _phonon(c):
    return c.frozen_phonon(S.fcc_au(6, 6, 1), 64, 64, 2, 3.0, 300.0, 1.2e7, -600.0, 1.5, nconfig=2, sigma=0.08, seed=3)[0]


def _jobs(c):
    jobs = []
    for j in range(6):
        n = (64, 128)[j % 2]
        d = dict(trans=_t(2, n), ax=0.1 * n, by=0.1 * n, kev=200.0, dz=[1.5, 1.6], layer_seq=[0, 1, 0])
        if j % 3 == 0:
            d["probe"] = (1.0, 0.05 * n, 0.05 * n)
        jobs.append(d)
    return np.concatenate([w.ravel() for w in c.run_jobs(jobs)])


def _scan(n):
    def run(c):
        det = [(0.2, 0.9), (1.0, 3.0)]
        return c.stem_scan(_t(1, n), 1.5, [0, 0], 0.06 * n, 0.06 * n, 200.0, 1.0, [[10.0, 10.0]], det, checkpoints=[0, 1])
    return run


def _transmission(c):
    v = np.random.default_rng(1).uniform(0, 300, (2, 64, 256)).astype(np.float32)
    return c.transmission(v, 6.0, 24.0, 200.0)


def _exit(c):
    return c.stem_exit_waves(_t(1, 128), 1.5, [0, 0], 8.0, 8.0, 200.0, 1.0, [[4.0, 4.0], [2.0, 3.0]])


CALLS = dict(multislice=_multislice, thick=_thick, image=_image, partial=_partial, potential=_potential,
             species=_species, phonon=_phonon, jobs=_jobs, scan_384=_scan(384), scan_768=_scan(768),
             transmission=_transmission, exit=_exit)
# bytes
LEAST = dict(multislice=268288, thick=6792192, jobs=1363216, scan_384=3712592, transmission=398336, exit=552992,
             potential=82928, species=153680, phonon=289340, image=591872, partial=756296, scan_768=14797904)


@pytest.mark.parametrize("call", sorted(CALLS))
def test_runs_in_the_cap_it_always_ran_in(call):
    from multislice_gb300 import Context
    with Context(0) as c:
        free = CALLS[call](c)
    with Context(0) as c:
        c.set_memory_limit(LEAST[call])
        assert np.array_equal(CALLS[call](c), free)
        assert c.memory_in_use() <= LEAST[call]


def test_a_cap_gives_the_image_buffer_back():
    """Images are summed up to 512 MB at a time without a cap; the buffer that takes
    does not stand in the way of a cap set later."""
    from multislice_gb300 import Context
    n, cap = 512, 64 << 20
    with Context(0) as c:
        c.ctem_image(_t(1, n), 1.5, [0], 30.0, 30.0, 200.0, 1.2e7, -600.0, 1.5, batch=16, df_spread=8.0, df_step=20.0)
        assert c.memory_in_use() > cap
        c.set_memory_limit(cap)
        assert c.memory_in_use() <= cap
        v = c.potential(S.srtio3(8, 8, 4), n, n, 2, 3.0)
        assert np.isfinite(v).all() and c.memory_in_use() <= cap
