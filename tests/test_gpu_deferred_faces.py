"""FP64 faces that leave the ordinary range go to a second pass over the
block's list of them: none, some and all faces of a block, in every tile
variant (their lists lie in different places), against the oracle bit for bit."""
import numpy as np
import pytest

from gpu_util import assert_bitwise, dev, host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def bsn():
    import bsn as b
    yield b
    b.set_tma(True)
    b.set_tile("f64", -1)


@pytest.mark.parametrize("share", [0.0, 0.02, 0.5, 1.0])
@pytest.mark.parametrize("n", [(32, 16, 16), (35, 17, 9)])
def test_deferred_faces_in_every_tile(orc, bsn, n, share):
    rng = np.random.default_rng(11)
    U = orc.state(*n)
    shape = U.shape[1:]
    U[0] = rng.uniform(0.5, 2.0, shape)
    for q in (1, 2, 3):
        U[q] = rng.uniform(-1.0, 1.0, shape)
    U[4] = rng.uniform(0.5, 2.0, shape) + 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / U[0]
    odd = rng.random(shape) < share          # cells beyond 2^116: their faces are deferred
    U[:, odd] *= 2.0 ** 130
    g, d = 5.0 / 3.0, 0.1
    dt = orc.cfl_dt_3d(U, d, d, d, g, 0.3)
    U0 = dev(U.copy(order="F"))
    for _ in range(2):
        orc.euler3d_step(U, d, d, d, dt, g)
    for tma in (True, False):
        bsn.set_tma(tma)
        for v in range(bsn.tile_variants("f64")):
            bsn.set_tile("f64", v)
            W = U0.clone()
            for _ in range(2):
                bsn.euler3d_step(W, *n, d, d, d, dt, g)
            assert_bitwise(host(W), U, f"tile {v}, TMA {tma}, share {share}")
