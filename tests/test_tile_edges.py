"""The fp64 and mixed builds' own flux kernels (2D x sweep + y runs, 1D line
tiles) and the register form of the block temperature solve against the
strict build's general kernels, at the edges of their tiles and segments:
axes below, at and above the 128-cell y segments, the sweep segments, the
line tiles (32 cells, above 18944 cells 122; in one-launch runs 32, above 14208
cells 58, above 25752 122, up to 54168; on 148 SMs), and the 512-cell register
slots of a block.

The flux bound is relative to dt/dx max(|F| + alpha |U|) of each field, the
size of the terms whose difference is taken: about 100 roundings of float64
(1e-13) and of float32 (2e-5) per face value, weights included."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

ND = {"P0": 10 * 101325, "T0": 300, "R0": 369, "x0": 0.08}
KEYS = ("left_boundary", "right_boundary", "bottom_boundary", "top_boundary")
BCS = {"walls": ("slip_wall", "zero_gradient", "slip_wall", "no_slip_wall"),
       "outlets": ("pressure_outlet", "no_slip_wall", "zero_gradient", "pressure_outlet"),
       "ends": ("pressure_outlet", "pressure_outlet"),  # 1D
       "ring": ("periodic", "periodic", "periodic", "periodic"),
       "injector": ("periodic", "periodic", "rdc_injector", "pressure_outlet")}


def _state(s, shape, nd=False, seed=5):
    """A jump in the middle of every axis, waves and 1 % of noise."""
    rng = np.random.default_rng(seed)
    full = (1,) + shape
    ax = np.meshgrid(*[np.arange(n) / n for n in shape], indexing="ij")
    hot = sum(a > 0.45 for a in ax) / len(shape)
    wave = 0.05 * sum(np.sin(5 * a + k) for k, a in enumerate(ax))
    P = (1.0 + 8.0 * hot + wave) * (1 + 0.01 * rng.uniform(-1, 1, shape))
    T = (1.2 + 5.0 * hot + wave) * (1 + 0.01 * rng.uniform(-1, 1, shape))
    if nd:
        P, T = P * 0.08, T
    else:
        P, T = P * 101325.0, T * 300.0
    Y = rng.uniform(0.0, 0.1, (8,) + shape)
    cu = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    c = 1.0 if nd else 300.0
    vel = [cu((c * (0.4 * hot + rng.uniform(-0.2, 0.2, shape))).reshape(full)) for _ in shape]
    return s.state_from_PTY(cu(P.reshape(full)), cu(T.reshape(full)), cu(Y), vel)


def _pair(dim, nx, ny, bc, prec, nd, d):
    from janc_b200 import mechanism as jm
    from janc_b200.solver import Solver
    mech = jm.load(jm.DEFAULT_MECHANISM, ND if nd else None)
    b = dict(zip(KEYS[: 2 * dim], BCS[bc]))
    mk = lambda p: Solver(dim, nx, ny if dim == 2 else None, d, d if dim == 2 else None, b, mech,  # noqa: E731
                          precision=p)
    return mk("fp64_strict"), mk(prec)


def _check_flux(s0, s1, U, aux, theta, d, prec):
    dt = 1e-8
    a, b = s0.flux_func(U, aux, dt=dt, theta=theta), s1.flux_func(U, aux, dt=dt, theta=theta)
    prim = s0.u_to_prim(U, aux)
    p, c = prim[-2], prim[-1]
    speed = sum(v.abs() for v in prim[1:1 + s0.dim]) + c
    tol = 1e-13 if prec == "fp64" else 2e-5
    for f in range(s0.nv):
        scale = float((speed * (U[f:f + 1].abs())).max())
        if f <= s0.dim:
            scale += float(p.max())
        if f == s0.dim + 1:
            scale += float((speed * p).max())
        assert float((a[f] - b[f]).abs().max()) <= tol * dt / d * scale, f
    assert s1.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,bc", [(4, 4, "walls"), (7, 31, "outlets"), (13, 127, "ring"), (6, 128, "walls"),
                                      (9, 129, "injector"), (5, 131, "outlets"), (50, 257, "walls"),
                                      (97, 6, "injector"), (61, 255, "ring")])
def test_sweep_flux_matches_the_strict_tiles(nx, ny, bc, prec):
    nd = bc == "injector"
    d = 0.0025 if nd else 1e-4
    s0, s1 = _pair(2, nx, ny, bc, prec, nd, d)
    U, aux = _state(s0, (nx, ny), nd)
    theta = {"Pb": 0.1 if nd else 101325.0}
    if nd:
        theta["Yinj"] = np.concatenate([[0.028, 0.22], 1e-20 * np.ones(6)])
    _check_flux(s0, s1, U, aux, theta if bc in ("outlets", "injector") else None, d, prec)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,bc", [(4, "ring"), (31, "walls"), (32, "outlets"), (33, "ends"), (34, "ends"),
                                   (64, "ring"), (65, "walls"), (18944, "outlets"), (18945, "walls"), (19031, "ends"),
                                   (19032, "ring"), (19033, "ends"), (19034, "ends"), (19067, "ring")])
def test_line_flux_matches_the_strict_tiles(nx, bc, prec):
    """One tile to both sides of the rule's line, and last tiles of one, two, all
    but one and all cells beside an outlet in either tile."""
    s0, s1 = _pair(1, nx, 1, bc, prec, False, 5e-5)
    U, aux = _state(s0, (nx,))
    _check_flux(s0, s1, U, aux, {"Pb": 101325.0} if bc in ("outlets", "ends") else None, 5e-5, prec)


@pytest.mark.gpu
@pytest.mark.parametrize("X,Y", [(7, 7), (16, 32), (19, 27), (32, 32), (41, 25), (44, 35), (45, 45), (46, 46)])
def test_block_update_matches_the_strict_loop(X, Y):
    """update_aux of blocks of 49 .. 2116 cells (one to four cells a thread,
    and the general loop above), guesses 20 % off.  Both stop when the block's
    largest residual is within 5e-9 J/kg, so T agrees within 2 * 5e-9 / cv and
    its rounding: 1e-12 relative."""
    from janc_b200.solver import Solver
    d = 1e-4
    s0 = Solver(2, 32, 32, d, d, precision="fp64_strict")
    s1 = Solver(2, 32, 32, d, d, precision="fp64")
    U, aux = _state(s0, (3 * X, Y))
    rng = np.random.default_rng(2)
    blk = lambda a: a.reshape(a.shape[0], 3, X, Y).transpose(0, 1).contiguous()  # noqa: E731
    Ub, ab = blk(U), blk(aux)
    guess = ab.clone()
    guess[:, 1] *= torch.as_tensor(rng.uniform(0.8, 1.2, (3, X, Y)), device="cuda")
    r0, r1 = s0.amr_update_aux(Ub, guess), s1.amr_update_aux(Ub, guess)
    assert float(((r1 - r0).abs() / r0.abs()).max()) <= 1e-12
    assert s1.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,bc", [(4, "ring"), (32, "ends"), (33, "ends"), (34, "ends"), (65, "ends"), (66, "ends"),
                                   (131, "walls"), (1301, "ring"), (11545, "ends"), (14208, "walls"), (14209, "ends"),
                                   (14211, "ends"), (20001, "ring"), (20012, "ends"), (25752, "walls"), (25753, "ends"),
                                   (25865, "ends"), (25866, "ends"), (54168, "walls")])
def test_line_run_is_the_separate_launches(nx, bc, prec):
    """advance of a 1D line as one persistent launch, bitwise the same steps
    as one launch per phase (the form that per-kernel timing takes): last
    tiles of one and two cells beside an outlet (33, 14211, 25865; 34, 20012,
    25866), one block, both sides of the tile sizes' limits, CFL and fixed
    steps, the launch repeated on its own workspace."""
    from janc_b200 import mechanism as jm
    from janc_b200.solver import Solver
    b = dict(zip(KEYS[:2], BCS[bc]))
    one, sep = [Solver(1, nx, dx=5e-5, boundary_config=b, mechanism=jm.load(), precision=prec) for _ in range(2)]
    sep.set_kernel_timing(True)
    U, aux = _state(one, (nx,))
    theta = {"Pb": 101325.0} if bc == "ends" else None
    for how in ({"cfl": 0.05}, {"dt": 1e-9}, {"cfl": 0.02}):
        a = one.advance(U, aux, 3, theta=theta, **how)
        r = sep.advance(U, aux, 3, theta=theta, **how)
        for x, y in zip(a, r):
            assert torch.equal(x, y) and bool(torch.isfinite(x).all())
    assert one.status() == sep.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nx", [20, 500, 14208, 14209, 25752, 25753, 54168])
def test_abandoned_line_run_shows_in_its_results(nx, prec):
    """A run whose first wait runs out (it expects a block that is never
    launched; one block, several, and every tile size to its limits) returns
    with NaN in place of the state and the time steps and with the status bit,
    and the same handle's next run is as if nothing had been.  So lines of
    these sizes do take the one launch."""
    from janc_b200 import _native
    from janc_b200 import mechanism as jm
    from janc_b200.solver import Solver
    b = dict(zip(KEYS[:2], BCS["walls"]))
    one, sep = [Solver(1, nx, dx=5e-5, boundary_config=b, mechanism=jm.load(), precision=prec) for _ in range(2)]
    sep.set_kernel_timing(True)
    U, aux = _state(one, (nx,))
    keep = U.clone(), aux.clone()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _native.check(one._lib.jb_selftest_line_run(one._h, 20.0, 1, 0, 0, st), one._h, "jb_selftest_line_run")
    for t in one.advance(U, aux, 3, cfl=0.05):
        assert bool(torch.isnan(t).all())
    assert one.status() == 16 and _native.status_text(16) == "device wait timed out"
    assert torch.equal(U, keep[0]) and torch.equal(aux, keep[1])
    for x, y in zip(one.advance(U, aux, 3, cfl=0.05), sep.advance(U, aux, 3, cfl=0.05)):
        assert torch.equal(x, y) and bool(torch.isfinite(x).all())
    assert one.status() == sep.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("before", [1, 17, 40, 100])
def test_line_run_barriers_count_past_32_bits(before, prec):
    """A run whose arrival count passes 2^32 (`before` arrivals into it: within
    a barrier, at one and between two of its 16 blocks' barriers) is the run
    that starts from zero, bit for bit."""
    from janc_b200 import _native
    from janc_b200 import mechanism as jm
    from janc_b200.solver import Solver
    s = Solver(1, 500, dx=5e-5, boundary_config=dict(zip(KEYS[:2], BCS["walls"])), mechanism=jm.load(), precision=prec)
    U, aux = _state(s, (500,))
    ref = s.advance(U, aux, 3, cfl=0.05)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _native.check(s._lib.jb_selftest_line_run(s._h, 1000.0, 0, 2 ** 32 - before, 0, st), s._h, "jb_selftest_line_run")
    for x, y in zip(s.advance(U, aux, 3, cfl=0.05), ref):
        assert torch.equal(x, y) and bool(torch.isfinite(x).all())
    assert s.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_refused_line_run_takes_the_separate_launches(prec):
    """A cooperative launch that the driver refuses (70000 cells are 574 blocks
    of the longest tiles, more than the device holds at three an SM) leaves the
    steps to the separate launches, and no error behind."""
    from janc_b200 import _native
    from janc_b200 import mechanism as jm
    from janc_b200.solver import Solver
    nx = 70000
    one, sep = [Solver(1, nx, dx=5e-5, boundary_config=dict(zip(KEYS[:2], BCS["walls"])), mechanism=jm.load(),
                       precision=prec) for _ in range(2)]
    U, aux = _state(one, (nx,))
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _native.check(one._lib.jb_selftest_line_run(one._h, 1000.0, 0, 0, 1, st), one._h, "jb_selftest_line_run")
    for x, y in zip(one.advance(U, aux, 2, cfl=0.05), sep.advance(U, aux, 2, cfl=0.05)):
        assert torch.equal(x, y) and bool(torch.isfinite(x).all())
    assert one.status() == sep.status() == 0


def test_arrival_counts_compare_modulo_2_to_32(tmp_path):
    """jb_arrived as the barriers use it, compiled for the host: a block whose
    target has wrapped waits for the arrivals before the wrap, and one whose
    target has not passes on a count that has."""
    src = tmp_path / "a.c"
    src.write_text('#include "jb_types.h"\nint arrived(unsigned c, unsigned t) { return jb_arrived(c, t); }\n')
    so = tmp_path / "a.so"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run(["gcc", "-shared", "-fPIC", "-I", os.path.join(root, "janc_b200", "csrc"), str(src), "-o", str(so)],
                   check=True)
    arrived = ctypes.CDLL(str(so)).arrived
    arrived.argtypes = [ctypes.c_uint, ctypes.c_uint]
    for base in (0, 444 * 7, 2 ** 31 - 100, 2 ** 32 - 500, 2 ** 32 - 1):
        target = (base + 444) % 2 ** 32
        for k in (0, 1, 443, 444, 445, 887):
            assert bool(arrived((base + k) % 2 ** 32, target)) == (k >= 444), (base, k)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(4, 4), (4, 8), (5, 7), (11, 3 * 32), (111, 128), (111, 129)])
def test_chemistry_forms_match_the_strict_build(nx, ny):
    """reaction_source_terms with four threads a cell (up to 14208 cells:
    whole and ragged 32-cell blocks, the largest of its range) and with one (the
    first size above), against the strict build's table-driven kernel; hot
    and cold cells, so both eliminations.  Two float64 evaluations of the rates,
    whose differences of near-equal rates amplify 1e-16 by up to 1e4."""
    s0, s1 = _pair(2, nx, ny, "walls", "fp64", False, 1e-4)
    U, aux = _state(s0, (nx, ny))
    a, b = s0.reaction_source_terms(U, aux, 3e-9), s1.reaction_source_terms(U, aux, 3e-9)
    for f in range(4, 12):
        assert float((a[f] - b[f]).abs().sum()) <= 1e-12 * float(a[f].abs().sum()), f
    assert s0.status() == s1.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("bx,by", [(1, 1), (1, 9), (5, 33), (20, 20), (21, 20), (24, 24), (40, 17)])
def test_block_stage_matches_the_strict_build(bx, by):
    """Stages of blocks whose interiors are one tile and several, one cell wide
    and ragged.  Each stage combines the state with dt L(U), both builds'
    fluxes within 1e-13 of the size of their terms: 1e-12 of each field."""
    from janc_b200.solver import Solver
    d, X, Y = 1e-4, bx + 6, by + 6
    s0 = Solver(2, 32, 32, d, d, precision="fp64_strict")
    s1 = Solver(2, 32, 32, d, d, precision="fp64")
    U, aux = _state(s0, (2 * X, Y))
    G = torch.cat([U, aux]).reshape(14, 2, X, Y).transpose(0, 1).contiguous()
    for stage in (1, 2, 3):
        a, b = (s.amr_stage(G, G if stage > 1 else None, stage, d, d, 1e-9) for s in (s0, s1))
        for f in range(14):
            assert float((a[:, f] - b[:, f]).abs().max()) <= 1e-12 * float(a[:, f].abs().max()), (stage, f)
    assert s0.status() == s1.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_grid_that_fits_without_the_sweep_scratch(prec):
    """A handle whose sweep scratch (24 bytes a cell) does not fit the device
    any more is made without it and takes the tile kernels: the strict build's
    fluxes and steps all the same.  Torch holds the rest of the memory
    meanwhile, but for what such a handle takes and half of the scratch."""
    from janc_b200 import mechanism as jm
    from janc_b200.solver import Solver
    nx, ny, d = 1024, 1024, 1e-4
    b = dict(zip(KEYS, BCS["walls"]))
    mk = lambda p: Solver(2, nx, ny, d, d, b, jm.load(), precision=p)  # noqa: E731
    s0 = mk("fp64_strict")
    U, aux = _state(s0, (nx, ny))
    ref = s0.advance(U, aux, 1, dt=1e-9)
    whole = mk(prec)
    bytes_whole = whole._lib.jb_workspace_bytes(whole._h)
    del whole
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    keep = bytes_whole - 12 * nx * ny
    fill = [torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")]
    try:
        s1 = mk(prec)
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    assert s1._lib.jb_workspace_bytes(s1._h) == bytes_whole - 24 * nx * ny
    _check_flux(s0, s1, U, aux, None, d, prec)
    for x, y in zip(s1.advance(U, aux, 1, dt=1e-9)[:2], ref[:2]):
        for f in range(x.shape[0]):
            tol = 1e-11 if prec == "fp64" else 1e-4
            assert float((x[f] - y[f]).abs().sum()) <= tol * float(y[f].abs().sum()), f
    assert s1.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["range", "mantissas", "edges"])
def test_reciprocal_is_within_two_ulp(kind):
    """rcp_nr, which the fast builds take for pivots, concentrations,
    equilibrium factors, Halley steps and float64 WENO weights, against 1 / x
    (correctly rounded): random numbers over all exponents whose reciprocal is
    normal, mantissas next to 1, 2 and the approximation's own steps, and the
    ends of the range; of 0, infinity and NaN it is NaN."""
    from janc_b200 import _native
    rng = np.random.default_rng(11)
    n = 1 << 20
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "range":
        x = sign * np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1020, 1021, n))
    elif kind == "mantissas":
        at = 1.0 + rng.integers(0, 1 << 20, n) * 2.0 ** -20  # a step of the 20-bit approximation
        x = sign * np.ldexp(np.nextafter(at, rng.choice([0.0, 3.0], n)), rng.integers(-40, 41, n))
        x[:3] = 1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0)
    else:
        x = np.repeat([2.0 ** -1021, 2.0 ** -1021 * (1 + 2.0 ** -52), 1e-300, 1e300, 2.0 ** 1021], 7)
    y = torch.empty(x.size, dtype=torch.float64, device="cuda")
    xd = torch.as_tensor(x, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    L = _native.lib()
    assert L.jb_probe_rcp(x.size, p(xd), p(y), st) == 0
    ref = 1.0 / x
    assert np.all(np.abs(y.cpu().numpy() - ref) <= 2.0 * np.spacing(np.abs(ref)))
    bad = torch.tensor([0.0, np.inf, -np.inf, np.nan], dtype=torch.float64, device="cuda")
    out = torch.empty_like(bad)
    assert L.jb_probe_rcp(4, p(bad), p(out), st) == 0
    assert bool(torch.isnan(out).all())
