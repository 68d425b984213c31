"""How one context's calls bear on one another: the tile a call takes, what it
launches and what it allocates do not depend on the calls before it."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import NG

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

G, DX, CFL = 5.0 / 3.0, 0.02, 0.4
KW = dict(rho_floor=1e-6, P_floor=1e-12)


@pytest.fixture(scope="module")
def bsn():
    import bsn as b
    yield b
    b.set_profiling(False)
    for p in ("f64", "f32", "learned"):
        b.set_tile(p, -1)


def _calm(bsn, n):
    """Uniform gas at rest around a small rough patch."""
    U = bsn.state(*n)
    U[0], U[4] = 1.0, 1.0 / (G - 1)
    p = (slice(NG + 20, NG + 30),) * 3
    r = torch.rand(10, 10, 10, generator=torch.Generator().manual_seed(3), dtype=torch.float64).cuda()
    U[(0,) + p] += r
    U[(4,) + p] += r
    return U


def _launches(bsn, names, f):
    bsn.set_profiling(True)
    f()
    got = [bsn.kernel_time(k)[1] for k in names]
    bsn.set_profiling(False)
    return got


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("first", ["nothing", "rhs", "stage", "step"])
def test_uniform_tiles_whatever_came_first(bsn, prec, first):
    """A right-hand side or a stage of the same grid cannot list uniform
    tiles; its tile choice is not the steps', nor the other way round."""
    n, dt = (128, 128, 128), 1e-3
    rhs, step = ((bsn.euler3d_rhs, bsn.euler3d_step) if prec == "f64"
                 else (bsn.euler3d_rhs_f32, bsn.euler3d_step_f32))
    U, V, F = _calm(bsn, n), bsn.state(*n), bsn.flux_arrays(*n)
    calls = {"rhs": lambda: rhs(V, *F, U, *n, DX, DX, DX, G, **KW),
             "stage": lambda: bsn.euler3d_stage(V, U, U, *n, DX, DX, DX, dt, G, 1, precision=prec, **KW),
             "step": lambda: step(U, *n, DX, DX, DX, dt, G, **KW), "nothing": lambda: None}
    bsn.set_tile(prec, -1)
    calls[first]()
    calls["step"]()
    assert _launches(bsn, ["uniform_stage_kernel"], calls["step"]) == [3]
    if first != "nothing":
        name = "stage_kernel" if prec == "f64" else "stage_kernel_f32"
        calls["rhs"]()
        assert _launches(bsn, ["uniform_stage_kernel"], calls["rhs"]) == [0]
        assert sum(_launches(bsn, [name, name + "_tma"], calls["rhs"])) == 1


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_reported_staging_is_the_one_that_runs(bsn, prec):
    n = (64, 64, 64)
    step = bsn.euler3d_step if prec == "f64" else bsn.euler3d_step_f32
    name = "stage_kernel_tma" if prec == "f64" else "stage_kernel_f32_tma"
    U = _calm(bsn, n)
    for tma in (True, False):
        bsn.set_tma(tma)
        for v in range(bsn.tile_variants(prec)):
            bsn.set_tile(prec, v)
            k, = _launches(bsn, [name], lambda: step(U, *n, DX, DX, DX, 1e-3, G, **KW))
            assert bsn.get_tile_tma(*n, prec) == (k > 0), (tma, v, k)
    bsn.set_tma(True)
    bsn.set_tile(prec, -1)


def test_step_captured_on_a_grid_not_seen_before(bsn):
    """A program that captures a step after another call has sized the
    workspace (a longer, thinner grid, too small for uniform tiles): the
    capture neither times tiles nor allocates."""
    from bsn._lib import load
    L = load()
    n, warm, dt = (64, 64, 64), (16, 16, 1000), 1e-3
    U = _calm(bsn, n)
    ref = U.clone()
    bsn.euler3d_step(ref, *n, DX, DX, DX, dt, G, **KW)
    W = bsn.state(*warm)
    W[0], W[4] = 1.0, 1.0 / (G - 1)
    s, ctx = torch.cuda.Stream(), C.c_void_p()
    torch.cuda.synchronize()
    assert L.bsn_ctx_create(C.byref(ctx), 0, C.c_void_p(s.cuda_stream)) == 0
    try:
        def step(A, m):
            return L.bsn_euler3d_step_f64(ctx, C.c_void_p(A.data_ptr()), *m, DX, DX, DX, dt, G, 0, KW["rho_floor"],
                                          KW["P_floor"])
        assert step(W, warm) == 0
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            rc = step(U, n)
        assert rc == 0, L.bsn_last_error(ctx).decode()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(U, ref)
        del g
    finally:
        torch.cuda.synchronize()
        L.bsn_ctx_destroy(ctx)


def test_captured_step_outlives_a_step_on_another_grid(bsn):
    """A captured step holds the workspace's addresses: a later step on a grid
    with more tiles, which the stage buffers have room for, moves none of it."""
    from bsn._lib import load
    L = load()
    dt = 1e-3
    n, other, room = (64, 64, 64), (72, 72, 72), (16, 16, 1000)
    U, V, W = _calm(bsn, n), _calm(bsn, other), bsn.state(*room)
    W[0], W[4] = 1.0, 1.0 / (G - 1)
    ref = U.clone()
    for _ in range(2):
        bsn.euler3d_step(ref, *n, DX, DX, DX, dt, G, **KW)
    s, ctx = torch.cuda.Stream(), C.c_void_p()
    torch.cuda.synchronize()
    assert L.bsn_ctx_create(C.byref(ctx), 0, C.c_void_p(s.cuda_stream)) == 0
    try:
        def step(A, m):
            rc = L.bsn_euler3d_step_f64(ctx, C.c_void_p(A.data_ptr()), *m, DX, DX, DX, dt, G, 0, KW["rho_floor"],
                                        KW["P_floor"])
            assert rc == 0, L.bsn_last_error(ctx).decode()
        assert L.bsn_ctx_set_tile(ctx, 0, 1) == 0     # forced: lists the tiles that are not uniform
        step(W, room)
        step(U, n)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            step(U, n)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        step(V, other)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(U, ref)
        del g
    finally:
        torch.cuda.synchronize()
        L.bsn_ctx_destroy(ctx)


def test_two_level_loop_takes_no_more_memory_than_its_levels(bsn):
    """The loop's workspace: two stage buffers a level, the coarse state before
    the step, the fine ghosts, and the registers of the coarse-fine faces; the
    tile choice is timed in them."""
    from bsn._lib import load
    L = load()
    m = 128
    U = _calm(bsn, (m, m, m))
    H = bsn.FMRGrid3D(U, m, m, m, DX, 33, 96, 33, 96, 33, 96, 2, G, **KW)
    bsn.fmr3d_run_steps(H, CFL, n_steps=1)     # loads the kernels
    ctx = C.c_void_p()
    torch.cuda.synchronize()
    assert L.bsn_ctx_create(C.byref(ctx), 0, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    try:
        t, k = C.c_double(0.0), C.c_int(0)
        free = torch.cuda.mem_get_info()[0]
        assert L.bsn_fmr3d_run_steps(ctx, C.byref(H.s), CFL, 1, 0, 1.0, 1, 0.0, C.byref(t), C.byref(k)) == 0
        torch.cuda.synchronize()
        state, faces = 5 * 8 * (m + 6) ** 3, 5 * 8 * 6 * m * m
        # allocations are rounded up to 2 MiB each; well under one more state
        assert free - torch.cuda.mem_get_info()[0] < 6 * state + 4 * faces + 8 * (2 << 20)
    finally:
        torch.cuda.synchronize()
        L.bsn_ctx_destroy(ctx)


def _loops(bsn, prec):
    """The device loops on a small grid: {name: (state tensors, advance by n
    steps from time t -> (t, steps))}."""
    m, out = 16, {}
    gen = torch.Generator().manual_seed(5)

    def gas(k):
        U = bsn.state(k, k, k)
        U[0] = 1.0 + 0.2 * torch.rand(U.shape[1:], generator=gen, dtype=torch.float64).cuda()
        U[4] = 2.0 * U[0]
        return U
    U = gas(m)
    out["run"] = ([U], lambda n, t: bsn.run_steps(U, m, m, m, DX, DX, DX, G, CFL, n_steps=n, t=t, precision=prec, **KW))
    V = gas(m)
    bhs = [bsn.BlackHole((0.05, 0.0, 0.0), (0.0, 0.3, 0.0), 0.1, 2 * DX, 1e6, 4 * DX)]
    out["coupled"] = ([V], lambda n, t: bsn.coupled_run_steps(V, bhs, m, m, m, DX, -8 * DX, -8 * DX, -8 * DX, G, CFL,
                                                              n_steps=n, t=t, self_gravity=True, precision=prec, **KW))
    H = bsn.FMRGrid3D(gas(m), m, m, m, DX, 5, 12, 5, 12, 5, 12, 2, G, **KW)
    out["two levels"] = ([H.Uc, H.Uf], lambda n, t: bsn.fmr3d_run_steps(H, CFL, n_steps=n, t=t, precision=prec))
    box = (5, 12, 5, 12, 5, 12, 2)
    N = bsn.FMRHierarchy3D(gas(m), m, m, m, DX, (box, box), G, **KW)
    out["levels"] = (list(N.levels), lambda n, t: bsn.fmr_nested_run_steps(N, CFL, n_steps=n, t=t, precision=prec))
    B = bsn.FMRHierarchy3D(gas(m), m, m, m, DX, (box, box), G, **KW)
    bh2 = [bsn.BlackHole((0.01, 0.0, 0.0), (0.0, 0.3, 0.0), 0.1, DX, 1e6, DX)]
    out["nested"] = (list(B.levels), lambda n, t: bsn.coupled_nested_run_steps(B, bh2, -8 * DX, -8 * DX, -8 * DX, CFL,
                                                                               n_steps=n, t=t, precision=prec))
    return out, (U, H, N, B), (bhs, bh2)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_short_calls_equal_one_long_call(bsn, prec):
    """One step a call (the first launched directly, the second captured, the
    rest replayed), a call of one length between those of another, and all
    steps in one call."""
    bsn.set_tile(prec, 0)
    loops, keep, holes = _loops(bsn, prec)
    bh0 = [[bytes(b) for b in h] for h in holes]
    start = {k: [a.clone() for a in s] for k, (s, _) in loops.items()}
    got = {}
    for name, (arrays, advance) in loops.items():
        for calls in ((7,), (1,) * 7, (1, 1, 3, 2), (2, 2, 1, 1, 1)):
            for a, b in zip(arrays, start[name]):
                a.copy_(b)
            for h, v in zip(holes, bh0):
                for b, raw in zip(h, v):
                    C.memmove(C.addressof(b), raw, len(raw))
            t, done = 0.0, 0
            for n in calls:
                t, k = advance(n, t)
                done += k
            torch.cuda.synchronize()
            res = [a.clone() for a in arrays]
            if name in got:
                assert (t, done) == got[name][0], (name, calls)
                assert all(torch.equal(x, y) for x, y in zip(res, got[name][1])), (name, calls)
            got[name] = ((t, done), res)
    bsn.set_tile(prec, -1)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_right_hand_side_times_its_own_tiles(bsn, prec):
    """A right-hand side stores fluxes and has another best tile than a stage:
    the first one on a grid times the tiles, whatever stage came before."""
    n = (40, 24, 24)
    rhs = bsn.euler3d_rhs if prec == "f64" else bsn.euler3d_rhs_f32
    U, V, F = bsn.state(*n), bsn.state(*n), bsn.flux_arrays(*n)
    U[0], U[4] = 1.0, 1.0 / (G - 1)
    bsn.set_tile(prec, -1)
    bsn.euler3d_stage(V, U, U, *n, DX, DX, DX, 1e-3, G, 1, precision=prec, **KW)
    counts = [bsn.launch_count()]
    for _ in range(3):
        rhs(V, *F, U, *n, DX, DX, DX, G, **KW)
        counts.append(bsn.launch_count())
    first, second, third = np.diff(counts)
    assert second == third and first > second + bsn.tile_variants(prec)


def _rough(bsn, n):
    """No uniform gas anywhere."""
    U = bsn.state(*n)
    w = 0.0
    for ax, m in enumerate(U.shape[1:]):
        x = torch.arange(m, device="cuda", dtype=torch.float64) * (2 * np.pi * (ax + 1) / (m - 2 * NG))
        w = w + torch.sin(x).reshape([-1 if a == ax else 1 for a in range(3)])
    U[0], U[4] = 1.0 + 0.2 * w, 2.0 + 0.4 * w
    return U


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_listing_follows_the_state(bsn, prec):
    """Steps and loops that listed uniform tiles stop when the state has none
    left, and take it up again, with the same bits throughout."""
    n, dt = (128, 128, 128), 1e-4
    step = bsn.euler3d_step if prec == "f64" else bsn.euler3d_step_f32
    calm, rough = _calm(bsn, n), _rough(bsn, n)
    a = (slice(None),) + (slice(NG, -NG),) * 3
    bsn.set_tile(prec, 0)
    want = {}
    for name, U0 in (("calm", calm), ("rough", rough)):
        U = U0.clone()
        step(U, *n, DX, DX, DX, dt, G, bc="periodic", **KW)
        V = U0.clone()
        bsn.run_steps(V, *n, DX, DX, DX, G, CFL, n_steps=2, bc="periodic", precision=prec, **KW)
        want[name] = U, V
    bsn.set_tile(prec, -1)
    for name, U0, times, listed in (("calm", calm, 2, 3), ("rough", rough, 20, 0), ("calm", calm, 80, 3)):
        for _ in range(times):
            U = U0.clone()
            step(U, *n, DX, DX, DX, dt, G, bc="periodic", **KW)
            assert torch.equal(U[a], want[name][0][a])
        U = U0.clone()
        k, = _launches(bsn, ["uniform_stage_kernel"],
                       lambda: step(U, *n, DX, DX, DX, dt, G, bc="periodic", **KW))
        assert k == listed, name

    def loop(U0, steps):
        U = U0.clone()
        c = bsn.launch_count()
        bsn.run_steps(U, *n, DX, DX, DX, G, CFL, n_steps=steps, bc="periodic", precision=prec, **KW)
        return U, bsn.launch_count() - c
    bsn.set_tile(prec, -1)
    per = {}
    for name, U0, times in (("calm", calm, 4), ("rough", rough, 4), ("calm", calm, 12)):
        for _ in range(times):
            U, c = loop(U0, 2)
            assert torch.equal(U[a], want[name][1][a])
        per[name] = c
    assert per["calm"] > per["rough"]          # a list takes a launch more per stage
    # one long call that starts on the list and goes on without it
    a_step = (loop(calm, 6)[1] - loop(calm, 2)[1]) / 4
    long, c = loop(rough, 300)
    assert c < 300 * a_step - 3 * 100
    U = rough.clone()
    t = 0.0
    for _ in range(3):
        t, _k = bsn.run_steps(U, *n, DX, DX, DX, G, CFL, n_steps=100, t=t, bc="periodic", precision=prec, **KW)
    assert torch.equal(U[a], long[a])
    bsn.set_tile(prec, -1)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("share", [0.3, 0.6, 0.85])
def test_listing_is_steady_on_one_state(bsn, prec, share):
    """Whether a list pays was timed on this state: steps that start from it
    again and again do not change sides, whatever share of it is uniform."""
    n = (150, 101, 67)
    step = bsn.euler3d_step if prec == "f64" else bsn.euler3d_step_f32
    U0 = _rough(bsn, n)
    k = NG + int(n[1] * (1 - share))
    U0[:, :, k:-NG] = 0.0
    U0[0, :, k:-NG], U0[4, :, k:-NG] = 1.0, 2.0
    U, seen = U0.clone(), set()
    bsn.set_tile(prec, -1)

    def one():
        U.copy_(U0)
        step(U, *n, DX, DX, DX, 1e-4, G, bc="periodic", **KW)
    for _ in range(8):
        one()
        seen.add((_launches(bsn, ["uniform_stage_kernel"], one)[0], bsn.get_tile(*n, prec)))
        for _ in range(12):
            one()
    assert len(seen) == 1, seen
    bsn.set_tile(prec, -1)
