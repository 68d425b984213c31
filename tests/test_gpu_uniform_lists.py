"""Uniform tiles through every tile variant (a forced one lists the tiles that
are not uniform), in the three precisions: single steps, and device loops,
which keep the tiles' flags from stage to stage and from step to step, both as
plain launches and as a captured graph.  Everything must have the bits of the
three stages with every face computed (euler3d_stage on caller-filled ghosts).
Sizes leave narrow last tiles; the state has uniform regions that meet inside
tiles, moving gas, gas too cold for the shortcut, a rough patch across a
periodic boundary and a ripple that FP32 cannot see."""
import numpy as np
import pytest

from gpu_util import NG
from test_gpu_floored_ghosts import _fill

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KW = dict(rho_floor=1e-6, P_floor=1e-12)
G, DX, CFL = 5.0 / 3.0, 0.02, 0.4
N = (97, 50, 58)


@pytest.fixture(scope="module")
def bsn():
    import bsn as b
    from bsn import learned
    learned.install(*learned.load_params())
    yield b
    for p in ("f64", "f32", "learned"):
        b.set_tile(p, -1)


def _state(bsn):
    rng = np.random.default_rng(9)
    W = np.empty((5,) + N)

    def put(sl, rho, v, P):
        W[(0,) + sl] = rho
        for q in range(3):
            W[(q + 1,) + sl] = rho * v[q]
        W[(4,) + sl] = P / (G - 1) + 0.5 * rho * sum(a * a for a in v)
    put((slice(None),) * 3, 1.0, (0.0, 0.0, 0.0), 1e-5)
    put((slice(45, None), slice(None), slice(20, None)), 0.7, (0.3, -0.2, 0.1), 2.0)
    put((slice(0, 20), slice(29, None), slice(0, 40)), 1e-3, (50.0, 0.0, 0.0), 1e-11)
    p = (slice(-3, None), slice(0, 9), slice(21, 30))
    W[(0,) + p] = rng.uniform(0.5, 2.0, W[(0,) + p].shape)
    W[(4,) + p] = rng.uniform(3.0, 5.0, W[(4,) + p].shape)
    p = (slice(20, 40), slice(0, 24), slice(0, 24))
    W[(0,) + p] *= 1.0 + 1e-12 * rng.uniform(-1.0, 1.0, W[(0,) + p].shape)
    U = bsn.state(*N)
    U[:, NG:-NG, NG:-NG, NG:-NG] = torch.from_numpy(W).cuda()
    return U


def _by_faces(bsn, U, dt, bc, prec):
    W, A, B = U.clone(), bsn.state(*N), bsn.state(*N)
    for s, (out, src) in enumerate(((A, W), (B, A), (W, B))):
        _fill(src, bc)
        bsn.euler3d_stage(out, src, W, *N, DX, DX, DX, dt, G, s + 1, precision=prec, **KW)
    return W


@pytest.mark.parametrize("bc", ["outflow", "periodic"])
@pytest.mark.parametrize("prec", ["f64", "f32", "learned"])
def test_steps_and_loops_equal_every_face_computed(bsn, bc, prec):
    step = {"f64": bsn.euler3d_step, "f32": bsn.euler3d_step_f32, "learned": bsn.euler3d_step_learned}[prec]
    steps = 7
    a = (slice(None),) + (slice(NG, -NG),) * 3
    bsn.set_tile(prec, -1)
    ref, ts, dts = [_state(bsn)], [0.0], []
    for _ in range(steps):
        dts.append(bsn.cfl_dt_3d(ref[-1], *N, DX, DX, DX, G, CFL))
        ts.append(ts[-1] + dts[-1])
        ref.append(_by_faces(bsn, ref[-1], dts[-1], bc, prec))
    for v in range(bsn.tile_variants(prec)):
        bsn.set_tile(prec, v)
        U = ref[0].clone()
        for k in range(3):
            step(U, *N, DX, DX, DX, dts[k], G, bc=bc, **KW)
            assert torch.equal(U[a], ref[k + 1][a]), (v, "step", k)
        for n in (1, 3, steps):
            U = ref[0].clone()
            got = bsn.run_steps(U, *N, DX, DX, DX, G, CFL, n_steps=n, bc=bc, precision=prec, **KW)
            assert got == (ts[n], n)
            assert torch.equal(U[a], ref[n][a]), (v, "loop", n)
    bsn.set_tile(prec, -1)


def test_choices_mixed_on_one_context(bsn):
    """Tiles and precisions that change between calls, and a right-hand side
    and a stage of the same grid before and between the steps."""
    a = (slice(None),) + (slice(NG, -NG),) * 3
    for p in ("f64", "f32", "learned"):
        bsn.set_tile(p, -1)
    U0, dU, F = _state(bsn), bsn.state(*N), bsn.flux_arrays(*N)
    dt = bsn.cfl_dt_3d(U0, *N, DX, DX, DX, G, CFL)
    step = {"f64": bsn.euler3d_step, "f32": bsn.euler3d_step_f32, "learned": bsn.euler3d_step_learned}
    ref = {p: _by_faces(bsn, U0, dt, "periodic", p) for p in step}
    bsn.euler3d_rhs(dU, *F, U0.clone(), *N, DX, DX, DX, G, bc="periodic", **KW)
    for p, v in (("f64", -1), ("f32", -1), ("f64", 1), ("learned", -1), ("learned", 3), ("f32", 2), ("f64", -1),
                 ("f32", -1), ("learned", -1)):
        bsn.set_tile(p, v)
        for q in step:
            U = U0.clone()
            step[q](U, *N, DX, DX, DX, dt, G, bc="periodic", **KW)
            assert torch.equal(U[a], ref[q][a]), (p, v, q)
    for p in step:
        bsn.set_tile(p, -1)
