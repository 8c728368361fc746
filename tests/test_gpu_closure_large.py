"""The closure on batches beyond one launch dimension's 65535 blocks, and on so many
pixels that a weight gradient's float sums would grow with the batch."""
import numpy as np
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


def _layers():
    """Slices of the parameter vector per layer: 1 -> 32 -> ... -> 32 -> 1 complex channels, 3 x 3 taps and biases."""
    o, out = 0, []
    for l in range(6):
        ci, co = (1 if l == 0 else 32), (1 if l == 5 else 32)
        out.append(slice(o, o + 9 * ci * co * 2 + co * 2))
        o = out[-1].stop
    return out


def test_weight_gradients_of_a_large_batch(ctx):
    """256 flat images of 512^2 against one of 128^2, whose sums are short.  The network
    divides a wave by its norm over 256^2 pixels, so the large images' inputs are a
    quarter of the small one's; with the first layer's weights and the targets scaled by
    4 every activation and, with the mean over 2^26 or 2^14 pixels, every gradient is the
    same but for powers of 2.  What differs is the error of the float sums, whose terms
    all have one sign: on the tensor cores (layers 1 to 4) at most an ulp (2^-23) of the
    running value, half the final one on average, per product of 16 pixels, 1024 of them
    for 16384 pixels; on the CUDA cores (layers 0 and 5) half an ulp per pixel, 8200 of
    them.  A parameter's gradient is a sum or difference of two such sums: sqrt 2."""
    from multislice_gb300.api import Closure
    net = Closure(ctx, seed=5)
    p = net.get_params()
    first = slice(0, 9 * 32 * 2)  # the first layer's weights

    def flat(b, n, z):
        return torch.full((b, n, n), z, dtype=torch.complex64, device="cuda")

    small = flat(1, 128, 0.75 + 0.5j), flat(1, 128, 0.6875 + 0.75j)   # target - wave = -0.0625 + 0.25i
    large = flat(256, 512, 0.75 + 0.5j), flat(256, 512, 0.5 + 1.5j)   # four times that
    torch.cuda.synchronize()
    q = p.copy()
    q[first] /= 4
    net.set_params(q)
    loss, ref = net.gradients(*small)
    ref[first] /= 4
    net.set_params(p)
    lossl, got = net.gradients(*large)
    net.close()
    del large
    torch.cuda.empty_cache()
    assert abs(lossl - loss) <= 1e-6 * loss
    for l, sl in enumerate(_layers()):
        tol = 2 ** 0.5 * (8200 * 2.0 ** -25 if l in (0, 5) else 1024 * 2.0 ** -24)
        d = got[sl].astype(np.float64) - ref[sl]
        err = np.linalg.norm(d) / np.linalg.norm(ref[sl])
        print("layer", l, err, tol)
        assert err < tol, l


@pytest.mark.parametrize("images,rows", [(1, 15), (1, 16), (1, 17), (2, 16), (3, 11), (1, 47)])
def test_weight_gradients_in_pieces(ctx, images, rows):
    """`images` flat images of `rows` rows an SM, whose sums are read out every 16 rows,
    against half the batch: the same gradient (the mean's factor 2 is exact) but for the
    two sums' errors, each at most 128 products' of 2^-24 and the read-outs' of 2^-24."""
    from multislice_gb300.api import Closure
    net = Closure(ctx, seed=9)
    b = 2 * (images * torch.cuda.get_device_properties(0).multi_processor_count // 2)
    c = torch.full((b, rows, 128), 0.75 + 0.5j, dtype=torch.complex64, device="cuda")
    f = torch.full((b, rows, 128), 0.5 + 1.5j, dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()
    loss, got = net.gradients(c, f)
    lossh, half = net.gradients(c[: b // 2], f[: b // 2])
    net.close()
    assert abs(loss - lossh) <= 1e-6 * lossh
    for l, sl in enumerate(_layers()):
        if 1 <= l <= 4:
            err = np.linalg.norm(got[sl].astype(np.float64) - half[sl]) / np.linalg.norm(half[sl])
            assert err < 2 * 2 ** 0.5 * (128 + 3) * 2.0 ** -24, l
