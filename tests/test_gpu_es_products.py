"""The early-stop network's products where their tiles (128 x 64 x 16), slices
and row ends can go wrong, against the FP64 CPU oracle on the same BF16 weights.
Tolerances as in the network's other oracle test: FP32 sums of up to some
thousand terms stay within 1e-4 (outputs) and 2e-3 (gradients, which pass
ReLUs) of the largest value."""
import numpy as np
import pytest

import es_net_oracle as O
from conftest import load_package

pkg = load_package()
from special_topics_b200 import earlystop as ES  # noqa: E402

pytestmark = pytest.mark.gpu


def _arch(length, convs, ch, k, stride, mlps, width):
    return dict(in_channels=2, in_length=length, conv_layers=convs, channels=ch, kernel=k, stride=stride,
                mlp_layers=mlps, mlp_width=width)


@pytest.mark.parametrize("arch,out_dim,B", [
    (_arch(33, 2, 7, 3, 3, 1, 65), 5, 1),        # nothing a multiple of four; one sample
    (_arch(33, 2, 7, 3, 3, 1, 65), 5, 129),      # one row past a tile
    (_arch(17, 1, 65, 7, 1, 2, 129), 1, 3),      # a column past a tile, kernel wider than the rest of a row
    (_arch(64, 2, 64, 5, 2, 1, 128), 64, 128),   # whole tiles
    (_arch(200, 1, 3, 5, 4, 1, 300), 2, 256),    # stride near the kernel, many slices of few values
    (_arch(9, 1, 1, 1, 1, 1, 1), 1, 2),          # smallest
])
def test_products_match_oracle(arch, out_dim, B):
    rng = np.random.default_rng(11)
    with ES.EsNet(out_dim, max_batch=256, **arch) as net:
        net.init(5)
        p = net.params
        x = rng.standard_normal((B, arch["in_length"], 2)).astype(np.float32)
        t = rng.standard_normal((B, out_dim)).astype(np.float32)
        w = rng.uniform(0.5, 2.0, out_dim).astype(np.float32)
        y = net.forward(x)
        yo, _ = O.forward(arch, out_dim, p, x)
        assert np.abs(y - yo).max() <= 1e-4 * np.abs(yo).max() + 1e-6
        loss, g = net.loss_grad(x, t, w)
        lo, go = O.loss_grad(arch, out_dim, p, x, t, w)
        assert abs(loss - lo) <= 1e-4 * lo
        for L in O.layers(arch, out_dim):
            for key in ("w", "b"):
                off, shape = L[key]
                sl = slice(off, off + int(np.prod(shape)))
                assert np.abs(g[sl] - go[sl]).max() <= 2e-3 * np.abs(go[sl]).max() + 1e-9, (key, off)
        assert np.array_equal(y[:1], net.forward(x[:1]))   # a sample's outputs do not depend on the others
