"""Kernels at the sizes where they can go wrong: tile edges, remainders, many contexts at once."""
import math

import numpy as np
import pytest

from helpers import oparams, source

pytestmark = pytest.mark.gpu


def test_ensemble_of_developed_members_matches_members_alone(engine):
    """Sixteen developed displacements whose kernels fill the GPU together end with the bits they
    have alone: no block may read a cell (the pinned one) that another block of its launch writes,
    since blocks start late when other members hold the SMs."""
    E = engine
    import torch

    def member(k):
        N = 128 * (1 + k % 4)
        P = E.default_params(N, N, stype=1, hmtype=4, nu=1.0, diffusion=1, alpha_l=1e-3, alpha_t=1e-4, eps=1e-8,
                             para_eps=1e-10, max_cycles=200, precision=1)
        ctx = E.Context(P)
        i = np.arange(N)
        r = np.hypot(i[:, None], i[None, :])
        c = np.zeros((N + 4, N + 4))
        c[2:-2, 2:-2] = 1.0 / (1.0 + np.exp((r - 0.35 * math.sqrt(2.0) * N) / 3.0))
        ctx.upload(c, source(oparams(P)), ghost=2)
        ctx.set_time(0.0)
        return ctx

    def state(ctx):
        N = ctx.P.N1
        c, p = np.zeros((N + 4, N + 4)), np.zeros((N + 4, N + 4))
        ctx.download(c, p, None, ghost=2)
        return c, p
    alone = []
    for k in range(16):
        ctx = member(k)
        ctx.step()
        alone.append(state(ctx))
        ctx.close()
    for _ in range(3):
        ens = E.Ensemble([member(k) for k in range(16)])
        ens.step(1)
        torch.cuda.synchronize()
        for ctx, (c, p) in zip(ens.members, alone):
            ce, pe = state(ctx)
            assert np.array_equal(ce, c) and np.array_equal(pe, p)
        ens.close()


@pytest.mark.parametrize("N1,N2", [(33, 65), (256, 256), (97, 70)])
@pytest.mark.parametrize("nu", [1.0, 2.0 / 3.0, 0.5])
@pytest.mark.parametrize("prec", [0, 1])
def test_cg_settles_at_its_floor(engine, oracle_lib, N1, N2, nu, prec):
    """A solve asked for more than FP64 gives ends near its best residual instead of drifting off
    from it: a mean in r or z must not reach CG's scalars.  The floor is the rounding of A x
    beside the wells, eps sum|a||x| per cell: below 1e-11 of ||f|| on these grids (the oracle's
    matrix confirms it).  The same fronts (M = 41) take at most 25 iterations to 1e-9."""
    import ctypes as C

    import torch

    import oracle as O
    from helpers import cell_ghost, dev, host
    E = engine
    i, j = np.arange(N1)[:, None], np.arange(N2)[None, :]
    wave = 1.0 + 0.2 * np.sin(0.3 * i) * np.cos(0.2 * j)
    c = 1.0 / (1.0 + np.exp((np.hypot(i, j) - 0.35 * wave * math.hypot(N1, N2)) / 2.0))
    for tol, cycles in ((1e-9, 25), (1e-16, 40)):
        P = E.default_params(N1, N2, stype=1, nu=nu, precision=prec, max_cycles=cycles)
        OP = oparams(P)
        q = source(OP)
        ctx = E.Context(P)
        ctx.set_source(dev(q))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        cyc, rr, status = ctx.pressure_solve(dev(c), p, tol, check=False)
        ctx.close()
        if tol == 1e-9:
            assert status == 0 and cyc <= cycles, (cyc, rr)
    A, b = np.zeros(N1 * N2 * 9), np.zeros(N1 * N2)
    oracle_lib.or_pressure_matrix(C.byref(OP), O.ptr(cell_ghost(OP, c)), O.ptr(A))
    oracle_lib.or_pressure_rhs(C.byref(OP), O.ptr(q), O.ptr(b))
    rr_or = oracle_lib.or_relres9(C.byref(OP), O.ptr(A), O.ptr(host(p).ravel().copy()), O.ptr(b))
    assert rr <= 1e-11 and rr_or <= 1e-11, (rr, rr_or)


@pytest.mark.parametrize("N1,N2", [(2, 2), (3, 33), (32, 32), (33, 31), (64, 34), (35, 97), (130, 36), (97, 161)])
@pytest.mark.parametrize("scheme", [4, 0, 1])  # MUSCL, upwind, WAF split
@pytest.mark.parametrize("mode", [4, 0, 1, 2, 3])
def test_sweep_tiles(engine, oracle_lib, N1, N2, scheme, mode):
    """The split sweeps at the edges of their 32 x 32 tiles (one cell over, one short, a last tile of
    one row, grids smaller than a halo) in every splitting, against the oracle.  A value is a
    sum of about 20 rounded terms of size <= 1 in either formulation: 1e-13."""
    import ctypes as C

    import oracle as O
    from helpers import cell_ghost, dev, host, rel_err, smooth_field, vel_split
    E = engine
    P = E.default_params(N1, N2, hmtype=scheme, dim_splitting=mode, porosity=0.7)
    OP = oparams(P)
    rng = np.random.default_rng(5)
    p = smooth_field(N1, N2, 9, -1.0, 1.0) * 0.05
    v = np.zeros(O.vel_shape(OP))
    c = rng.uniform(0.0, 1.0, (N1, N2))
    cg = cell_ghost(OP, c)
    oracle_lib.or_calc_velocities(C.byref(OP), O.ptr(cell_ghost(OP, p)), O.ptr(v), O.ptr(cg))
    u, vv = vel_split(OP, v)
    dt = 0.8 * oracle_lib.or_max_stable_advection_dt(C.byref(OP), O.ptr(v)) * OP.porosity
    pfs = C.c_int(1)
    oracle_lib.or_advect_split(C.byref(OP), O.ptr(cg), O.ptr(v), dt, C.byref(pfs))
    ctx = E.Context(P)
    d = dev(c)
    assert ctx.advect_split(d, dev(u), dev(vv), dt, 1) == pfs.value
    assert rel_err(host(d), O.interior(OP, cg)) <= 1e-13
    ctx.close()


@pytest.mark.parametrize("N1,N2", [(2, 2), (3, 5), (16, 32), (17, 33), (15, 31), (33, 257), (48, 513), (130, 70)])
@pytest.mark.parametrize("stype", [0, 2])  # wells; a Dirichlet row in the CN system (N1 >= 4)
def test_cn_half_step_at_tile_edges(engine, oracle_lib, N1, N2, stype):
    """The dispersion kernels at the edges of their 16 x 32 tiles, row segments (256 and 512
    columns) and odd row counts, against the oracle's CN solve.  Both stop at 1e-13 of ||b|| and
    the matrix is within a factor 3 of the identity here: 1e-12, in the norm that the residual has."""
    import ctypes as C

    import oracle as O
    from helpers import cell_ghost, dev, host, smooth_field, vel_split
    if stype == 2 and N1 < 4:
        return
    E = engine
    P = E.default_params(N1, N2, stype=stype, diffusion=1, alpha_l=0.5, alpha_t=0.05, Dm=1e-3, para_eps=1e-13, max_cycles=400)
    OP = oparams(P)
    v = np.zeros(O.vel_shape(OP))
    c = np.random.default_rng(6).uniform(0.0, 1.0, (N1, N2))
    cg = cell_ghost(OP, c)
    p = smooth_field(N1, N2, 9, -1.0, 1.0) * 0.05
    oracle_lib.or_calc_velocities(C.byref(OP), O.ptr(cell_ghost(OP, p)), O.ptr(v), O.ptr(cg))
    u, vv = vel_split(OP, v)
    dt = 0.5 * oracle_lib.or_max_stable_dt(C.byref(OP), O.ptr(v))
    its, rr = C.c_int(), C.c_double()
    assert oracle_lib.or_cn_solve(C.byref(OP), O.ptr(cg), O.ptr(v), dt, 0, 1e-14, C.byref(its), C.byref(rr)) == 0
    ctx = E.Context(P)
    d = dev(c)
    _, rr_d = ctx.dispersion_cn(d, dev(u), dev(vv), dt, 1e-13)
    assert rr_d <= 1e-13
    ref = O.interior(OP, cg)
    assert np.linalg.norm(host(d) - ref) <= 1e-12 * np.linalg.norm(ref)
    ctx.close()


@pytest.mark.parametrize("N1,N2", [(130, 132), (131, 257), (260, 130), (514, 515), (1030, 770)])
@pytest.mark.parametrize("prec", [0, 1])
def test_half_cycle_kernels_match_separate_launches(engine, monkeypatch, N1, N2, prec):
    """A half cycle per launch (tiles with a recomputed halo; 16-byte and element staging, last tiles
    of a few rows and columns) gives the bits of one launch per colour and transfer: the same
    cycles, residual and pressure.  A context without the red-black shortcuts runs the latter."""
    import torch

    from helpers import dev, host
    E = engine
    c = np.random.default_rng(4).uniform(0.0, 1.0, (N1, N2))
    out = []
    for skip in ("1", "0"):
        monkeypatch.setenv("IMPEC_MG_RB_SKIP", skip)
        P = E.default_params(N1, N2, stype=1, nu=1.0, precision=prec, max_cycles=200)
        ctx = E.Context(P)
        ctx.set_source(dev(source(oparams(P))))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        n0 = E.launch_count(ctx)
        cyc, rr, _ = ctx.pressure_solve(dev(c), p, 1e-10)
        out.append((cyc, rr, host(p), E.launch_count(ctx) - n0))
        ctx.close()
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])
    assert out[0][3] < out[1][3]


@pytest.mark.parametrize("N1,N2", [(1001, 900), (900, 1001), (100, 8004), (101, 8001), (8001, 100), (1500, 560), (887, 1122)])
def test_marching_half_cycles(engine, monkeypatch, N1, N2):
    """Large FP32 levels, a warp per strip and segment (16-byte and element copies, strips and segments of
    all remainders): the bits of one launch per colour and transfer."""
    import torch

    from helpers import dev, host
    E = engine
    c = np.random.default_rng(4).uniform(0.0, 1.0, (N1, N2))
    out = []
    for skip in ("1", "0"):
        monkeypatch.setenv("IMPEC_MG_RB_SKIP", skip)
        P = E.default_params(N1, N2, stype=1, nu=1.0, precision=1, max_cycles=200, x_lb=0.0, x_ub=float(N1), y_lb=0.0,
                             y_ub=float(N2))
        ctx = E.Context(P)
        ctx.set_source(dev(source(oparams(P))))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        cyc, rr, _ = ctx.pressure_solve(dev(c), p, 1e-10)
        out.append((cyc, rr, host(p)))
        ctx.close()
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("N1,N2", [(2, 1025), (2, 2000), (2000, 2), (3, 1300)])
@pytest.mark.parametrize("nu", [1.0, 0.25])
def test_thin_grids(engine, monkeypatch, N1, N2, nu):
    """Grids of a few rows have more levels below 1,024 cells than the single-CTA coarse cycle holds.
    Both precisions solve the same system to 1e-10 of ||f||; with square cells its condition number is
    of the order of max(N1, N2)^2 = 4e6, so the pressures agree to 1e-3."""
    import torch

    from helpers import dev, host
    E = engine
    monkeypatch.setenv("IMPEC_MG_CLUSTER", "0")
    out = []
    for prec in (0, 1):
        P = E.default_params(N1, N2, stype=1, nu=nu, precision=prec, max_cycles=200, x_lb=0.0, x_ub=float(N1), y_lb=0.0,
                             y_ub=float(N2))
        ctx = E.Context(P)
        ctx.set_source(dev(source(oparams(P))))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        rr = ctx.pressure_solve(dev(np.random.default_rng(8).uniform(0.0, 1.0, (N1, N2))), p, 1e-10)[1]
        assert rr <= 1e-10
        out.append(host(p))
        ctx.close()
    assert np.linalg.norm(out[0] - out[1]) <= 1e-3 * np.linalg.norm(out[0])


@pytest.mark.parametrize("N1,N2", [(2, 2), (3, 3), (5, 7), (31, 33), (127, 129), (517, 301), (1021, 1031)])
@pytest.mark.parametrize("prec", [0, 1])
def test_cg_vectors_in_pairs(engine, N1, N2, prec):
    """CG over odd and even cell counts, one and several pairs per thread.  The reported residual is
    recomputed from the iterate; the cycle's contraction (below 1/3) takes 1e-10 in some 20 iterations."""
    import torch

    from helpers import dev, host
    E = engine
    P = E.default_params(N1, N2, stype=1, nu=1.0, precision=prec, max_cycles=60)
    ctx = E.Context(P)
    c = dev(np.random.default_rng(8).uniform(0.0, 1.0, (N1, N2)))
    ctx.set_source(dev(source(oparams(P))))
    p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
    cyc, rr, _ = ctx.pressure_solve(c, p, 1e-10)
    assert rr <= 1e-10 and cyc <= 30
    assert np.isfinite(host(p)).all()
    ctx.close()


@pytest.mark.parametrize("B,H,W,cin,cout", [
    (1, 1, 1, 32, 32), (2, 3, 17, 32, 64), (3, 2, 63, 64, 32), (1, 5, 65, 8, 32), (2, 7, 100, 32, 8), (1, 130, 64, 96, 32),
    (5, 1, 129, 64, 64), (2, 33, 200, 128, 64), (7, 61, 70, 32, 32), (1, 2, 32, 64, 160), (64, 24, 24, 8, 8), (1, 300, 40, 64, 96)])
def test_weight_gradient_by_rows(engine, B, H, W, cin, cout):
    """Weight gradients by image rows: one and several strips, partial last strips, runs that end within
    and across strips and images, all box widths.  Against FP64 sums of the same bf16 inputs: products are
    exact and partial sums FP32, 2^-24 relative per addition, random over up to 8e4 terms: 2e-5 of the
    largest entry (entries are of the order of sqrt(terms) / 2)."""
    import ctypes as C

    import torch
    import torch.nn.functional as F
    E = engine
    L = E.lib()
    vp = lambda t: C.c_void_p(t.data_ptr())
    g = torch.Generator(device="cuda").manual_seed(B + W)
    X = torch.randn((B, H, W, cin), device="cuda", generator=g).to(torch.bfloat16)
    dZ = (torch.randn((B, H, W, cout), device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    Kp = (9 * cin + 63) // 64 * 64
    dW = torch.zeros((cout, Kp), device="cuda")
    assert L.impec_conv3x3_weight_grad(vp(dZ), vp(X), B, H, W, cin, cout, vp(dW), None) == 0, E.last_error()
    xp, dz = F.pad(X.double(), (0, 0, 1, 1, 1, 1)), dZ.double().reshape(-1, cout)
    ref = torch.zeros((cout, Kp), device="cuda", dtype=torch.float64)
    for tap in range(9):
        y, x = divmod(tap, 3)
        ref[:, tap * cin:(tap + 1) * cin] = dz.T @ xp[:, y:y + H, x:x + W].reshape(-1, cin)
    assert (dW.double() - ref).abs().max().item() <= 2e-5 * ref.abs().max().item()


@pytest.mark.parametrize("B,H,W", [(3, 8, 8), (2, 8, 72), (2, 40, 24)])
def test_net_gradients_of_batches(engine, B, H, W):
    """Pooling, upsampling and their gradients over batches and images that are not square: the gradients
    of a batch are the mean of its images' from the CPU restatement, with that comparison's tolerance
    (bf16 rounding of every stored activation)."""
    import torch

    from oracle import learned_ref as R
    E = engine
    net = E.Net(seed=3)
    g = torch.Generator(device="cuda").manual_seed(5)
    X = torch.zeros((B, H, W, 8), device="cuda")
    X[..., :4] = torch.randn((B, H, W, 4), generator=g, device="cuda")
    X = X.to(torch.bfloat16)
    T = torch.randn((B, H, W), generator=g, device="cuda")
    loss = net.backprop(X, T)
    grads, params = net.parameters(which=1), net.parameters(which=0)
    refs = [R.forward_backward(params, X[b].float().cpu().numpy(), T[b].cpu().numpy()) for b in range(B)]
    loss_ref, grads_ref = np.mean([r[0] for r in refs]), np.mean([r[1] for r in refs], axis=0)
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref)
    off = 0
    for cin, cout, *_ in R.LAYERS:
        n = cout * R.kp(cin) + cout
        a, b = grads[off:off + n], grads_ref[off:off + n]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b) + 1e-12
        off += n
    net.close()


@pytest.mark.parametrize("N1,N2", [(2, 2), (3, 257), (129, 65), (700, 513)])
def test_diagnostics_on_the_edges(engine, N1, N2):
    """Mass, flux through the boundary faces, extremes of both signs and a NaN that the extremes pass over:
    sums of at most 4e5 terms of the order of one, 1e-12 relative."""
    from helpers import dev
    E = engine
    ctx = E.Context(E.default_params(N1, N2, stype=1))
    rng = np.random.default_rng(N1)
    c, u, v = rng.normal(size=(N1, N2)), rng.normal(size=(N1 + 1, N2)), rng.normal(size=(N1, N2 + 1))
    be = np.abs(u[0]).sum() + np.abs(u[-1]).sum() + np.abs(v[:, 0]).sum() + np.abs(v[:, -1]).sum()
    d = ctx.diagnostics(dev(c), dev(u), dev(v))
    assert d[3] == c.max() and d[4] == c.min()
    assert abs(d[2] - be) <= 1e-12 * be
    for s in (1.0, -1.0):  # one sign only
        d = ctx.diagnostics(dev(s * np.abs(c)), dev(u), dev(v))
        assert d[3] == (s * np.abs(c)).max() and d[4] == (s * np.abs(c)).min()
    c[0, 0] = np.nan
    d = ctx.diagnostics(dev(c), dev(u), dev(v))
    assert d[3] == np.nanmax(c) and d[4] == np.nanmin(c)
    ctx.close()


@pytest.mark.parametrize("N1,N2", [(64, 64), (65, 130), (130, 300)])
@pytest.mark.parametrize("kind", ["inclusions", "closed", "barriers"])
@pytest.mark.parametrize("nu", [1.0, 2.0 / 3.0])
@pytest.mark.parametrize("prec", [0, 1])
def test_contrasts_inside_coarse_cells(engine, N1, N2, kind, nu, prec):
    """Nearly impermeable and impermeable inclusions, and thin barriers crossed by a channel: coarse cells
    that hold both sides of a contrast, on all levels.  CG in 64-bit numpy with these coarse operators takes 10
    to 12 iterations to 1e-9 on the five-point systems; twice as many are allowed for FP32 cycles and for the
    nine-point operator's condition number of 1 / nu."""
    import torch

    from helpers import dev
    E = engine
    i, j = np.arange(N1)[:, None], np.arange(N2)[None, :]
    K = np.ones((N1, N2))
    if kind == "barriers":
        K[N1 // 3, :N2 * 2 // 3] = 1e-8
        K[N1 // 5:N1 // 3, N2 // 2] = 1e-6
        K[:, N2 // 4] = 1e4
    else:
        K[np.sin(0.37 * i) * np.cos(0.29 * j) > 0.5] = 1e-10 if kind == "inclusions" else 0.0
        K[:3, :3] = K[-3:, -3:] = 1.0
    P = E.default_params(N1, N2, stype=1, nu=nu, precision=prec, max_cycles=24, x_lb=0.0, x_ub=float(N1), y_lb=0.0,
                         y_ub=float(N2))
    ctx = E.Context(P)
    ctx.set_source(dev(source(oparams(P))))
    ctx.set_permeability(dev(K), dev(K))
    p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
    cyc, rr, _ = ctx.pressure_solve(dev(np.zeros((N1, N2))), p, 1e-9)
    assert rr <= 1e-9, (cyc, rr)
    ctx.close()


@pytest.mark.parametrize("N1,N2,aniso", [(130, 900, 0.01), (96, 700, 0.02), (200, 200, 0.01)])
@pytest.mark.parametrize("nu", [1.0, 0.9])
@pytest.mark.parametrize("prec", [0, 1])
def test_cg_stays_at_its_floor_when_the_residual_is_replaced(engine, N1, N2, aniso, nu, prec):
    """A tolerance a little below what FP64 gives: the recurrence residual passes it again and again, and
    each time the true residual takes its place.  CG must go on from there, not from a search direction that
    belongs to the old residual: 400 iterations leave the residual within ten times of its floor (the smallest that
    solves of 60 to 160 iterations reach)."""
    import torch

    from helpers import dev
    E = engine
    i, j = np.arange(N1)[:, None], np.arange(N2)[None, :]
    K = np.exp(0.7 * np.sin(0.21 * i + 0.05 * j) * np.cos(0.17 * j))
    c = 1.0 / (1.0 + np.exp((np.hypot(i, j) - 0.35 * math.hypot(N1, N2)) / 3.0))

    def solve(tol, cycles):
        P = E.default_params(N1, N2, stype=1, nu=nu, precision=prec, max_cycles=cycles, x_lb=0.0, x_ub=float(N1), y_lb=0.0,
                             y_ub=float(N2))
        ctx = E.Context(P)
        ctx.set_source(dev(source(oparams(P))))
        ctx.set_permeability(dev(K), dev(aniso * K))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        rr = ctx.pressure_solve(dev(c), p, tol, check=False)[1]
        ctx.close()
        return rr
    floor = min(solve(1e-16, n) for n in (60, 90, 120, 160))
    for part in (0.9, 0.75, 0.6, 0.4):
        assert solve(part * floor, 400) <= 10.0 * floor, part


@pytest.mark.parametrize("N1,N2", [(2, 2048), (5, 2049), (3, 2561)])
def test_cn_sweep_on_few_long_rows(engine, oracle_lib, N1, N2):
    """Few long rows: each colour of a sweep is a launch of its own whose blocks share the rows (two launches more
    per sweep than on a short grid).  The same comparison as test_cn_half_step_at_tile_edges, for the same reasons."""
    import ctypes as C

    import oracle as O
    from helpers import cell_ghost, dev, host, smooth_field, vel_split
    E = engine

    def launches(N1, N2):
        P = E.default_params(N1, N2, diffusion=1, alpha_l=0.5, alpha_t=0.05, Dm=1e-3, para_eps=1e-13, max_cycles=400,
                             x_lb=0.0, x_ub=float(N1), y_lb=0.0, y_ub=float(N2))
        OP = oparams(P)
        v = np.zeros(O.vel_shape(OP))
        c = np.random.default_rng(6).uniform(0.0, 1.0, (N1, N2))
        cg = cell_ghost(OP, c)
        p = smooth_field(N1, N2, 9, -1.0, 1.0) * 0.05
        oracle_lib.or_calc_velocities(C.byref(OP), O.ptr(cell_ghost(OP, p)), O.ptr(v), O.ptr(cg))
        u, vv = vel_split(OP, v)
        dt = 0.5 * oracle_lib.or_max_stable_dt(C.byref(OP), O.ptr(v))
        its, rr = C.c_int(), C.c_double()
        assert oracle_lib.or_cn_solve(C.byref(OP), O.ptr(cg), O.ptr(v), dt, 0, 1e-14, C.byref(its), C.byref(rr)) == 0
        ctx = E.Context(P)
        d = dev(c)
        n0 = E.launch_count(ctx)
        sweeps, rr_d = ctx.dispersion_cn(d, dev(u), dev(vv), dt, 1e-13)
        n = E.launch_count(ctx) - n0
        ctx.close()
        ref = O.interior(OP, cg)
        assert rr_d <= 1e-13 and np.linalg.norm(host(d) - ref) <= 1e-12 * np.linalg.norm(ref)
        return n, sweeps
    n, sweeps = launches(N1, N2)
    m, short = launches(N1, 64)
    assert (n - 2) / sweeps == (m - 2) / short + 2  # beside the matrix and the right-hand side


@pytest.mark.parametrize("N1,N2,launches", [(4, 20000, 2), (5, 13200, 2), (6, 14000, 2), (8, 13000, 1), (33, 2010, 2), (40, 2500, 1),
                                            (24, 4100, 1), (7000, 24, 1)])
@pytest.mark.parametrize("scheme", [4, 1])  # MUSCL, WAF split
def test_sweeps_of_thin_grids(engine, oracle_lib, N1, N2, launches, scheme):
    """Grids of few rows: X, then Y cell by cell (two launches) where the tiles' rows would lie beyond the
    grid for the most part, else tiles of 8 rows; Strang, symmetric and single sweeps take the same rules.  Against the
    oracle, with the tolerance of test_sweep_tiles for its reasons (the single sweeps against each other: 1e-13 too)."""
    import ctypes as C

    import oracle as O
    from helpers import cell_ghost, dev, host, rel_err, smooth_field, vel_split
    E = engine
    c = np.random.default_rng(5).uniform(0.0, 1.0, (N1, N2))
    p = smooth_field(N1, N2, 9, -1.0, 1.0) * 0.05
    for mode in (1, 3, 4):  # X first, Strang, symmetric
        P = E.default_params(N1, N2, hmtype=scheme, dim_splitting=mode, porosity=0.7)
        OP = oparams(P)
        v = np.zeros(O.vel_shape(OP))
        cg = cell_ghost(OP, c)
        oracle_lib.or_calc_velocities(C.byref(OP), O.ptr(cell_ghost(OP, p)), O.ptr(v), O.ptr(cg))
        u, vv = vel_split(OP, v)
        dt = 0.8 * oracle_lib.or_max_stable_advection_dt(C.byref(OP), O.ptr(v)) * OP.porosity
        pfs = C.c_int(1)
        oracle_lib.or_advect_split(C.byref(OP), O.ptr(cg), O.ptr(v), dt, C.byref(pfs))
        ctx = E.Context(P)
        d = dev(c)
        n0 = E.launch_count(ctx)
        ctx.advect_split(d, dev(u), dev(vv), dt, 1)
        n = E.launch_count(ctx) - n0
        assert rel_err(host(d), O.interior(OP, cg)) <= 1e-13
        if mode == 1:
            assert n == launches
            s = dev(c)
            ctx.advect_x(s, dev(u), dt)
            ctx.advect_y(s, dev(vv), dt)
            assert rel_err(host(s), host(d)) <= 1e-13
        ctx.close()


@pytest.mark.parametrize("W", [3, 6, 7])
@pytest.mark.parametrize("cin,cout", [(8, 32), (32, 128), (256, 256)])
def test_weight_gradient_of_narrow_images(engine, W, cin, cout):
    """Either side of six columns, where the general kernel gives way to image rows.  The comparison of
    test_weight_gradient_by_rows, for its reasons."""
    test_weight_gradient_by_rows(engine, 48, 33, W, cin, cout)


@pytest.mark.parametrize("N1,N2", [(37, 29), (100, 100), (300, 130), (65, 257)])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("env", [{"IMPEC_MG_KRYLOV": "0"}, {"IMPEC_MG_RB_RESID": "0"}, {"IMPEC_MG_PRE": "0", "IMPEC_MG_POST": "2"},
                                 {"IMPEC_MG_KRYLOV": "0", "IMPEC_MG_RB_RESID": "0"}, {"IMPEC_MG_PRE": "2", "IMPEC_MG_POST": "0"}],
                         ids=["stationary", "all residuals", "no pre-smoothing", "stationary, all residuals", "no post-smoothing"])
def test_cluster_takes_every_schedule(engine, monkeypatch, N1, N2, prec, env):
    """Stationary cycles (plain transfers), restrictions that take both colours' residuals and one-sided smoothing run
    their coarse levels in the cluster launch too, with the bits of the per-level launches."""
    import torch

    from helpers import dev, host
    E = engine
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    c = np.random.default_rng(9).uniform(0.0, 1.0, (N1, N2))
    out = []
    for cluster in ("0", "1"):
        monkeypatch.setenv("IMPEC_MG_CLUSTER", cluster)
        P = E.default_params(N1, N2, stype=1, nu=1.0, precision=prec, max_cycles=200, x_lb=0.0, x_ub=float(N1), y_lb=0.0,
                             y_ub=float(N2))
        ctx = E.Context(P)
        ctx.set_source(dev(source(oparams(P))))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        n0 = E.launch_count(ctx)
        cyc, rr, _ = ctx.pressure_solve(dev(c), p, 1e-9, check=False)
        out.append((cyc, rr, host(p), E.launch_count(ctx) - n0))
        ctx.close()
    assert np.isfinite(out[0][1]) and out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])
    assert out[1][3] < out[0][3]


@pytest.mark.parametrize("nu,ok", [(1.0, True), (0.9, False), (0.5, False), (0.25, False)])
def test_cold_sweep_timing_is_for_five_point_systems(engine, nu, ok):
    """Nine-point systems are refused, whatever levels precondition them."""
    import ctypes as C

    import torch
    E = engine
    ctx = E.Context(E.default_params(96, 96, stype=1, nu=nu))
    flush = torch.zeros(1 << 20, device="cuda")
    ms, best, b = C.c_double(), C.c_double(), C.c_double()
    st = E.lib().impec_time_kernel_cold(ctx.h, 0, 1, C.c_void_p(flush.data_ptr()), flush.numel() * 4, C.byref(ms), C.byref(best),
                                        C.byref(b))
    assert (st == 0) == ok
    ctx.close()


@pytest.mark.parametrize("N1,N2,stype", [(300, 130, 1), (515, 333, 1), (97, 70, 2), (1024, 1024, 1)])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 1), (2, 1)])
def test_one_launch_sweeps_under_cg(engine, monkeypatch, N1, N2, stype, prec, pre, post):
    """The default schedule of a CG solve runs half cycles in one launch; with any other one the levels sweep by colour or, from
    the tile thresholds on, both colours in one launch (from x = 0 as well).  Either way the same bits."""
    import torch

    from helpers import dev, host
    E = engine
    monkeypatch.setenv("IMPEC_MG_PRE", str(pre))
    monkeypatch.setenv("IMPEC_MG_POST", str(post))
    c = np.random.default_rng(12).uniform(0.0, 1.0, (N1, N2))
    out = []
    for tile in ("0", "1"):
        monkeypatch.setenv("IMPEC_MG_TILE_CELLS", tile)
        monkeypatch.setenv("IMPEC_MG_TILE_CELLS32", tile)
        P = E.default_params(N1, N2, stype=stype, nu=1.0, precision=prec, max_cycles=200)
        ctx = E.Context(P)
        ctx.set_source(dev(source(oparams(P))))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        n0 = E.launch_count(ctx)
        cyc, rr, _ = ctx.pressure_solve(dev(c), p, 1e-10)
        out.append((cyc, rr, host(p), E.launch_count(ctx) - n0))
        ctx.close()
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])
    assert out[1][3] < out[0][3]


@pytest.mark.parametrize("N1,N2", [(33, 40), (3, 2100)])
def test_hyperbolic_solve_leaves_the_iterate_of_a_failed_dispersion_solve(engine, N1, N2):
    """A CN solve that does not converge ends the update; c holds the iterate it stopped at, the one that the
    dispersion entry point leaves for the same half step (without wells nothing precedes it): the same bits."""
    import torch

    from helpers import dev, host
    E = engine
    rng = np.random.default_rng(3)
    c, u, v = rng.uniform(0.0, 1.0, (N1, N2)), rng.normal(size=(N1 + 1, N2)), rng.normal(size=(N1, N2 + 1))
    P = E.default_params(N1, N2, diffusion=1, alpha_l=0.5, alpha_t=0.05, Dm=1e-3, para_eps=1e-30, max_cycles=2)
    out = []
    for call in ("hyperbolic_solve", "dispersion_cn"):
        ctx = E.Context(P)
        d, dt = dev(c), 1e-4
        with pytest.raises(E.ImpecError) as e:
            getattr(ctx, call)(d, dev(u), dev(v), dt if call == "hyperbolic_solve" else 0.5 * dt)
        torch.cuda.synchronize()
        out.append((e.value.status, host(d).copy()))
        ctx.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1]) and not np.array_equal(out[0][1], c)


@pytest.mark.parametrize("N1,N2,stype", [(515, 333, 1), (1024, 1024, 1), (600, 410, 2)])
def test_one_launch_sweeps_above_half_cycles(engine, monkeypatch, N1, N2, stype):
    """A finest FP64 level that streams from HBM sweeps in one launch while the levels below it run half cycles: the bits
    of half cycles throughout, from the host and from the captured solve."""
    import torch

    from helpers import dev, host
    E = engine
    c = np.random.default_rng(12).uniform(0.0, 1.0, (N1, N2))
    cg = np.zeros((N1 + 4, N2 + 4))
    cg[2:-2, 2:-2] = c
    out = []
    for tile in (0, N1 * N2):
        monkeypatch.setenv("IMPEC_MG_TILE_CELLS", str(tile))
        P = E.default_params(N1, N2, stype=stype, nu=1.0, precision=0, max_cycles=200, eps=1e-10)
        ctx = E.Context(P)
        q = source(oparams(P))
        ctx.set_source(dev(q))
        p = torch.zeros((N1, N2), dtype=torch.float64, device="cuda")
        n0 = E.launch_count(ctx)
        cyc, rr, _ = ctx.pressure_solve(dev(c), p, 1e-10)
        n = E.launch_count(ctx) - n0
        ctx.upload(cg, q, ghost=2)
        res = [ctx.pressure_solve_resident() for _ in range(3)]
        pr = np.zeros((N1 + 4, N2 + 4))
        ctx.download(None, pr, None, ghost=2)
        out.append((cyc, rr, host(p), res, pr, n))
        ctx.close()
    assert out[0][:2] == out[1][:2] and out[0][3] == out[1][3]
    assert np.array_equal(out[0][2], out[1][2]) and np.array_equal(out[0][4], out[1][4])
    assert out[1][5] > out[0][5]
