"""States below a floor beside the grid's boundary.  The scheme floors active
cells and takes ghost cells raw, so a floored cell differs from the ghosts
that were copied from it and the boundary faces carry a flux, however uniform
the gas is.  Steps through every tile variant (a forced one lists the tiles
that are not uniform) must give the bits of the three stages with every face
computed (euler3d_stage on caller-filled ghosts), and in FP64 the oracle's."""
import numpy as np
import pytest

from gpu_util import NG, dev, host

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KW = dict(rho_floor=1e-3, P_floor=2e-5)
G, DX, DT = 5.0 / 3.0, 0.02, 0.02


@pytest.fixture(scope="module")
def bsn():
    import bsn as b
    from bsn import learned
    learned.install(*learned.load_params())
    yield b
    for p in ("f64", "f32", "learned"):
        b.set_tile(p, -1)


def _state(orc, n, below):
    """Gas at rest: all of it below P_floor, all below rho_floor, or its lower
    half in z below P_floor."""
    U = orc.state(*n)
    # (a density below its floor comes with a pressure that pushes mass in from
    # the raw ghosts: from a cold or thinner gas every cell ends at the floors)
    U[0] = 1.0 if below != "rho" else 0.9 * KW["rho_floor"]
    P = np.full(U.shape[1:], 0.5 * KW["P_floor"] if below != "rho" else 1e-2)
    if below == "half":
        P[:, :, NG + n[2] // 2:] = 1e-3
    U[4] = P / (G - 1)
    return U


def _fill(U, bc):
    for ax in (1, 2, 3):
        m = U.shape[ax] - 2 * NG
        for g in range(NG):
            lo, hi = (NG, NG + m - 1) if bc == "outflow" else (g + m, g + NG)
            U.narrow(ax, g, 1).copy_(U.narrow(ax, lo, 1))
            U.narrow(ax, NG + m + g, 1).copy_(U.narrow(ax, hi, 1))


def _by_faces(bsn, U, n, bc, prec):
    """One step with every face computed."""
    W, A, B = U.clone(), bsn.state(*n), bsn.state(*n)
    for s, (out, src) in enumerate(((A, W), (B, A), (W, B))):
        _fill(src, bc)
        bsn.euler3d_stage(out, src, W, *n, DX, DX, DX, DT, G, s + 1, precision=prec, **KW)
    return W


@pytest.mark.parametrize("n", [(64, 64, 64), (97, 50, 58)])
@pytest.mark.parametrize("bc", ["outflow", "periodic"])
@pytest.mark.parametrize("below", ["P", "rho", "half"])
@pytest.mark.parametrize("prec", ["f64", "f32", "learned"])
def test_steps_from_below_a_floor(orc, bsn, n, bc, below, prec):
    step = {"f64": bsn.euler3d_step, "f32": bsn.euler3d_step_f32, "learned": bsn.euler3d_step_learned}[prec]
    U = _state(orc, n, below)
    U0 = dev(U)
    bsn.set_tile(prec, -1)
    ref = [U0]
    for _ in range(2):
        ref.append(_by_faces(bsn, ref[-1], n, bc, prec))
    a = (slice(None),) + (slice(NG, -NG),) * 3
    assert torch.unique(ref[1][a][0]).numel() > 1      # the boundary's flux shows
    if prec == "f64":
        orc.euler3d_step(U, DX, DX, DX, DT, G, bc=bc, **KW)
        assert np.array_equal(host(ref[1])[a], U[a])
    for v in range(bsn.tile_variants(prec)):
        bsn.set_tile(prec, v)
        W = U0.clone()
        for k in range(2):
            step(W, *n, DX, DX, DX, DT, G, bc=bc, **KW)
            assert torch.equal(W[a], ref[k + 1][a]), (v, k)
    bsn.set_tile(prec, -1)
