"""msl_stem_exit_waves into host memory, an aligned device buffer (where the slice loop
then runs), one the passes cannot take, and one that overlaps the transmission
functions: the same waves bit for bit."""
import numpy as np
import pytest

from multislice_gb300 import specimen as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _setup(n, nprobe):
    rng = np.random.default_rng(n)
    trans = np.exp(0.3j * rng.standard_normal((2, n, n))).astype(np.complex64)
    xy = rng.uniform(2.0, 18.0, (nprobe, 2))
    args = (1.7, [0, 1, 1], 20.0, 21.0, 200.0, float(S.mrad_to_k(25.0, 200.0)), xy)
    return trans, args


@pytest.mark.parametrize("n,batch", [(256, 4), (384, 3), (128, 0)])
def test_where_the_waves_go_does_not_change_them(n, batch):
    from multislice_gb300 import Context
    nprobe = 10  # a ragged last batch
    trans, args = _setup(n, nprobe)
    t = torch.from_numpy(trans).cuda()
    flat = torch.empty(nprobe * n * n + 2, dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    with Context(0) as c:
        c.set_probe_batch(batch)
        ref = c.stem_exit_waves(trans, *args)
        for shift in (0, 1):  # 16-byte aligned, 8 bytes off
            out = flat[shift:shift + nprobe * n * n].view(nprobe, n, n)
            c.stem_exit_waves(t, *args, out=out)
            assert np.array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("lead", [0, 1, 3])  # layers' worth of memory before the transmission functions
def test_output_over_the_transmission_functions(lead):
    from multislice_gb300 import Context
    n, nprobe = 128, 4
    trans, args = _setup(n, nprobe)
    flat = torch.empty((6, n, n), dtype=torch.complex64, device="cuda")
    with Context(0) as c:
        ref = c.stem_exit_waves(trans, *args)
        t = flat[lead:lead + 2]
        t.copy_(torch.from_numpy(trans))
        torch.cuda.synchronize()
        c.stem_exit_waves(t, *args, out=flat[:nprobe])
        assert np.array_equal(flat[:nprobe].cpu().numpy(), ref)
