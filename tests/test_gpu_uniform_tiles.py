"""Blocks of uniform gas skip their faces (stage_tile.cuh).  The steps must
give the bits of the composition that computes every face: euler3d_rhs! with
its flux arrays materialised (which never skips), the SSP-RK3 combinations
and the floors.  The state has several uniform regions meeting at odd places,
one of them too cold for the shortcut and one moving, and a rough patch that
crosses a periodic boundary; sizes leave narrow last tiles."""
import numpy as np
import pytest

from gpu_util import NG

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KW = dict(rho_floor=1e-6, P_floor=1e-12)
G, DX, DT = 5.0 / 3.0, 0.02, 2e-4


@pytest.fixture(scope="module")
def bsn():
    import bsn as b
    yield b
    for p in ("f64", "f32"):
        b.set_tile(p, -1)


def _state(bsn, n, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = n
    U = np.zeros((5,) + n)

    def put(sl, rho, v, P):
        U[(0,) + sl] = rho
        for q in range(3):
            U[(q + 1,) + sl] = rho * v[q]
        U[(4,) + sl] = P / (G - 1) + 0.5 * rho * sum(a * a for a in v)
    put((slice(None),) * 3, 1.0, (0.0, 0.0, 0.0), 1e-5)
    put((slice(33, None),) * 3, 0.7, (0.3, -0.2, 0.1), 2.0)             # moving
    put((slice(0, 20), slice(29, None), slice(0, 40)), 1e-3, (50.0, 0.0, 0.0), 1e-11)   # cold and fast
    p = (slice(-3, None), slice(0, 9), slice(21, 30))                    # rough, at a boundary
    U[(0,) + p] = rng.uniform(0.5, 2.0, U[(0,) + p].shape)
    U[(4,) + p] = rng.uniform(0.5, 2.0, U[(4,) + p].shape)
    D = bsn.state(*n)
    D[:, NG:-NG, NG:-NG, NG:-NG] = torch.from_numpy(U).cuda()
    return D


def _by_faces(bsn, U, n, bc, prec):
    """One step with every face computed."""
    rhs = bsn.euler3d_rhs if prec == "f64" else bsn.euler3d_rhs_f32
    F, dU, W, Un = bsn.flux_arrays(*n), bsn.state(*n), U.clone(), U.clone()
    for s in range(3):
        rhs(dU, *F, W, *n, DX, DX, DX, G, bc=bc, **KW)
        if s == 0:
            W.copy_(Un + DT * dU)
        elif s == 1:
            W.copy_((0.75 * Un + 0.25 * W) + (0.25 * DT) * dU)
        else:
            W.copy_(((1.0 / 3.0) * Un + (2.0 / 3.0) * W) + ((2.0 / 3.0) * DT) * dU)
        bsn.apply_floors_3d(W, *n, KW["rho_floor"], KW["P_floor"], G)
    return W


@pytest.mark.parametrize("n", [(64, 64, 64), (66, 65, 67), (97, 50, 58)])
@pytest.mark.parametrize("bc", ["outflow", "periodic"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_steps_equal_every_face_computed(bsn, n, bc, prec):
    step = bsn.euler3d_step if prec == "f64" else bsn.euler3d_step_f32
    U0 = _state(bsn, n, 3)
    ref = [U0]
    for _ in range(3):
        ref.append(_by_faces(bsn, ref[-1], n, bc, prec))
    a = (slice(None),) + (slice(NG, -NG),) * 3
    for v in [-1] + list(range(bsn.tile_variants(prec))):
        bsn.set_tile(prec, v)
        for tma in (True, False):
            bsn.set_tma(tma)
            U = U0.clone()
            for k in range(3):
                step(U, *n, DX, DX, DX, DT, G, bc=bc, **KW)
                assert torch.equal(U[a], ref[k + 1][a]), (v, tma, k)
    bsn.set_tma(True)
    bsn.set_tile(prec, -1)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_device_loop_equals_single_steps(bsn, prec):
    """The loop keeps the uniform tiles from one step to the next; single
    steps find them anew."""
    n = (97, 50, 58)
    step = bsn.euler3d_step if prec == "f64" else bsn.euler3d_step_f32
    U, V = _state(bsn, n, 4), _state(bsn, n, 4)
    t, k = bsn.run_steps(U, *n, DX, DX, DX, G, 0.4, n_steps=6, precision=prec, **KW)
    ts = 0.0
    for _ in range(6):
        dt = bsn.cfl_dt_3d(V, *n, DX, DX, DX, G, 0.4)
        step(V, *n, DX, DX, DX, dt, G, **KW)
        ts += dt
    assert (t, k) == (ts, 6)
    assert torch.equal(U, V)
