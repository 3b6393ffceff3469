"""GPU parity of the RHS and the RK4 time step against the CPU oracle and the
reference-generated golden fixtures (all calls go through the C ABI)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _to_dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.to(dtype)


def _fab_from_valid(A, valid, ng, dtype):
    c, nz, ny, nx = valid.shape
    t = A.new_fab((nx, ny, nz), ng, dtype=dtype, ncomp=c)
    A.valid(t, ng).copy_(_to_dev(valid, dtype))
    A.fill_periodic_ghosts(t, ng)
    return t


def _rel_max(a, b):
    """max over planes of max|a-b| / max|b| (per component)."""
    out = 0.0
    for c in range(a.shape[0]):
        scale = max(np.abs(b[c]).max(), 1e-300)
        out = max(out, np.abs(a[c] - b[c]).max() / scale)
    return out


@pytest.mark.parametrize("box", ["rand", "ic"])
def test_eval_rhs_f64_bit_exact_vs_reference(axs, golden, box):
    g = golden("fields_f64.npz")
    dx, kappa, lam, R2 = g["params"][:4]
    soln = _fab_from_valid(axs, g[f"{box}_state"], 2, torch.float64)
    c, nz, ny, nx = g[f"{box}_state"].shape
    rhs = axs.new_fab((nx, ny, nz), 0, dtype=torch.float64)
    coeffs = axs._lib.RhsCoeffs(kappa, lam, R2)
    axs.eval_rhs(soln, rhs, 2, 0, dx, coeffs)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(rhs.cpu().numpy(), g[f"{box}_rhs"])


@pytest.mark.parametrize("box", ["rand", "ic"])
def test_eval_rhs_f32_vs_reference_float_build(axs, golden, box):
    g = golden("fields_f32.npz")
    dx, kappa, lam, R2 = g["params"][:4]
    soln = _fab_from_valid(axs, g[f"{box}_state"], 2, torch.float32)
    c, nz, ny, nx = g[f"{box}_state"].shape
    rhs = axs.new_fab((nx, ny, nz), 1, dtype=torch.float32)
    axs.eval_rhs(soln, rhs, 2, 1, dx, axs._lib.RhsCoeffs(kappa, lam, R2))
    got = axs.valid(rhs, 1).cpu().numpy()
    ref = g[f"{box}_rhs"]
    np.testing.assert_array_equal(got[:2], ref[:2])  # rhs_psi = Pi exactly
    # FP32 arithmetic order differs from the FLOAT build's double-weight diff2: a few ulp of the stencil scale
    scale = np.abs(g[f"{box}_state"][:2]).max() * 16 / dx ** 2 * 3
    assert np.abs(got[2:] - ref[2:]).max() <= 4e-6 * scale


def test_fill_lincomb_combine(axs, orc):
    rng = np.random.default_rng(5)
    v = rng.standard_normal((4, 6, 7, 8))
    t = _fab_from_valid(axs, v, 2, torch.float64)
    f = orc.to_fab(v, 2)
    np.testing.assert_array_equal(t.cpu().numpy(), f)
    x = _fab_from_valid(axs, rng.standard_normal((4, 6, 7, 8)), 2, torch.float64)
    y = _fab_from_valid(axs, rng.standard_normal((4, 6, 7, 8)), 2, torch.float64)
    d = torch.zeros_like(x)
    axs.lincomb(d, x, 0.37, y, 2)
    xv, yv = axs.valid(x, 2).cpu().numpy(), axs.valid(y, 2).cpu().numpy()
    np.testing.assert_array_equal(axs.valid(d, 2).cpu().numpy(), xv + 0.37 * yv)  # no contraction
    ks = [_fab_from_valid(axs, rng.standard_normal((4, 6, 7, 8)), 2, torch.float64) for _ in range(4)]
    axs.rk4_combine(d, x, *ks, 2, 0.1)
    V = [axs.valid(k, 2).cpu().numpy() for k in ks]
    ref = axs.valid(x, 2).cpu().numpy() + (0.1 / 6) * (V[0] + 2 * V[1] + 2 * V[2] + V[3])
    np.testing.assert_array_equal(axs.valid(d, 2).cpu().numpy(), ref)


def _stagewise_rk4(axs, state_valid, dx, bg, tau_i, t0, dt, nsteps):
    """The drop-in path: per-stage specific_eval_rhs + LinComb, as GRTeclyn drives it."""
    ng = 2
    c, nz, ny, nx = state_valid.shape
    u = _fab_from_valid(axs, state_valid, ng, torch.float64)
    uold, us = torch.zeros_like(u), torch.zeros_like(u)
    ks = [torch.zeros_like(u) for _ in range(4)]
    lvl = axs.AxionStringsLevel((nx, ny, nz), dx, bg, tau_i=tau_i, dtype=torch.float64)
    t = t0
    for _ in range(nsteps):
        uold.copy_(u)
        for s, (ts, cs) in enumerate(((t, 0.5 * dt), (t + 0.5 * dt, 0.5 * dt), (t + 0.5 * dt, dt), (t + dt, None))):
            src = uold if s == 0 else us
            axs.fill_periodic_ghosts(src, ng)
            lvl.specific_eval_rhs(src, ks[s], ts, ng_soln=ng, ng_rhs=ng)
            if cs is not None:
                axs.lincomb(us, uold, cs, ks[s], ng)
        axs.rk4_combine(u, uold, *ks, ng, dt)
        t += dt
    return axs.valid(u, ng).cpu().numpy()


def test_stagewise_rk4_matches_oracle(axs, orc):
    rng = np.random.default_rng(11)
    v = rng.standard_normal((4, 10, 12, 16)) * np.array([1, 1, .3, .3])[:, None, None, None]
    dx, dt, n = 0.5, 0.1, 6
    bgo = orc.background(a_inv=1.5, c0=1.0, lambda_scale=2.0)
    fab = orc.to_fab(v, 2)
    orc.rk4_advance(fab, 2, dx, bgo, 1.0, 0.0, dt, n)
    ref = orc.from_fab(fab, 2)
    got = _stagewise_rk4(axs, v, dx, axs.Background.expanding(1.5, 1.0, lambda0=2.0), 1.0, 0.0, dt, n)
    # FP64 RHS and stage combinations evaluate the same expressions with the same
    # rounding as the CPU restatement: bit-exact
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("shape", [(16, 12, 10), (32, 20, 7), (48, 33, 16), (8, 4, 5), (4, 2, 3)])
def test_fused_rk4_f64_matches_oracle(axs, orc, shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + ny + nz)
    v = rng.standard_normal((4, nz, ny, nx)) * np.array([1, 1, .3, .3])[:, None, None, None]
    dx, dt, n = 0.5, 0.1, 12
    # matter domination (a_inv = 1.5): nonzero curvature term, time-dependent lambda -> stage times matter
    bgo = orc.background(a_inv=1.5, c0=1.0, lambda_scale=2.0)
    fab = orc.to_fab(v, 2)
    orc.rk4_advance(fab, 2, dx, bgo, 1.0, 0.0, dt, n)
    ref = orc.from_fab(fab, 2)
    lv = axs.PeriodicLevel((nx, ny, nz), dx, dtype=torch.float64)
    lv.set_state(_to_dev(v))
    lv.advance(axs.Background.expanding(1.5, 1.0, lambda0=2.0), 1.0, 0.0, dt, n)
    lv.device_status()
    got = lv.get_state().cpu().numpy()
    assert _rel_max(got, ref) < 1e-12


def test_fused_rk4_config_plain_64cubed_100_steps(axs, orc):
    """64^3, dx=0.5, dt=0.1, 100 steps, RD (a_inv=2), fat strings (c0=1), lambda0=2, FP64:
    fields within 1e-10 relative of the oracle."""
    n, dx, dt, steps = 64, 0.5, 0.1, 100
    v = orc.fourier_ic_state(n, orc.strict_cutoff(n / 4), seed=1234)
    bgo = orc.background(a_inv=2.0, c0=1.0, lambda_scale=2.0)
    fab = orc.to_fab(v, 2)
    orc.rk4_advance(fab, 2, dx, bgo, 1.0, 0.0, dt, steps)
    ref = orc.from_fab(fab, 2)
    lv = axs.PeriodicLevel(n, dx, dtype=torch.float64)
    lv.set_state(_to_dev(v))
    lv.advance(axs.Background.expanding(2.0, 1.0, lambda0=2.0), 1.0, 0.0, dt, steps)
    lv.device_status()
    got = lv.get_state().cpu().numpy()
    assert _rel_max(got, ref) < 1e-10


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 2e-5)])
def test_homogeneous_solution_is_exact(axs, dtype, tol):
    """psi = R(tau), Pi = R'(tau) solves the full EOM (test_background.cpp:69-89);
    in radiation domination R = tau is linear, which RK4 integrates exactly."""
    n, dx, dt, steps = 16, 0.5, 0.1, 40
    bg = axs.Background.expanding(2.0, 1.0, lambda0=2.0)
    v = torch.zeros((4, n, n, n), dtype=torch.float64)
    v[0] = bg.R(1.0)
    v[2] = bg.R_prime(1.0)
    lv = axs.PeriodicLevel(n, dx, dtype=dtype)
    lv.set_state(v.cuda())
    lv.advance(bg, 1.0, 0.0, dt, steps)
    s = lv.get_state().double().cpu()
    tau_f = 1.0 + steps * dt
    assert torch.allclose(s[0], torch.full_like(s[0], bg.R(tau_f)), rtol=tol, atol=0)
    assert torch.allclose(s[2], torch.full_like(s[2], bg.R_prime(tau_f)), rtol=tol, atol=tol)
    assert float(s[1].abs().max()) == 0.0 and float(s[3].abs().max()) == 0.0


def _check_padding(lv, val):
    """The 8 columns either side in x (whole 32-byte sectors; the stencils read 4)
    and 2 rows either side in y hold periodic copies (nx >= 8)."""
    st = lv.state.cpu().numpy()
    ox, oy, nx, ny = lv.layout.x_offset, lv.layout.y_offset, lv.nx, lv.ny
    rows = st[:, :, oy:oy + ny]
    np.testing.assert_array_equal(rows[..., ox - 8:ox], val[..., nx - 8:nx])
    np.testing.assert_array_equal(rows[..., ox + nx:ox + nx + 8], val[..., :8])
    np.testing.assert_array_equal(st[:, :, oy - 2:oy, ox:ox + nx], val[:, :, ny - 2:ny, :])
    np.testing.assert_array_equal(st[:, :, oy + ny:oy + ny + 2, ox:ox + nx], val[:, :, :2, :])


def test_level_fab_round_trip(axs):
    rng = np.random.default_rng(3)
    v = rng.standard_normal((4, 9, 10, 12))
    t = _fab_from_valid(axs, v, 3, torch.float64)
    lv = axs.PeriodicLevel((12, 10, 9), 0.5, dtype=torch.float64)
    lv.import_fab(t, 3)
    np.testing.assert_array_equal(lv.get_state().cpu().numpy(), v)
    out = axs.new_fab((12, 10, 9), 1, dtype=torch.float64)
    lv.export_fab(out, 1)
    np.testing.assert_array_equal(axs.valid(out, 1).cpu().numpy(), v)
    # padding holds periodic copies
    _check_padding(lv, v)


def test_fused_rk4_keeps_padding_current(axs):
    rng = np.random.default_rng(8)
    v = rng.standard_normal((4, 8, 6, 8)) * 0.5
    lv = axs.PeriodicLevel((8, 6, 8), 0.5, dtype=torch.float64)
    lv.set_state(_to_dev(v))
    lv.advance(axs.Background.flat(1.0), 0.0, 0.0, 0.05, 3)
    _check_padding(lv, lv.get_state().cpu().numpy())


def test_fused_rk4_f64_512cubed_matches_oracle(axs, orc):
    """The precision workload's grid in FP64 (512^3, dx 0.5, Moore c0 = 2,
    lambda0 = 2, RD, Fourier IC |n| < N/8), 2 steps, against the oracle's
    stage-by-stage RK4: element offsets past 32 bits on real 3-D data. The
    oracle holds about 40 GB on the host."""
    import os
    if os.sysconf("SC_PAGE_SIZE") * os.sysconf("SC_PHYS_PAGES") < 96 * 2 ** 30:
        pytest.skip("the 512^3 FP64 oracle needs about 40 GB of host memory")
    from axion_strings_adaptive_gb300 import ic
    n, dx, dt, steps = 512, 0.5, 0.1, 2
    s0 = ic.fourier_state(n, ic.strict_cutoff(n / 8), seed=31, dtype=torch.float64, device="cuda")
    lv = axs.PeriodicLevel(n, dx, dtype=torch.float64, pierced_capacity=1024)
    lv.set_state(s0)
    lv.advance(axs.Background.expanding(2.0, 2.0, lambda0=2.0), 1.0, 0.0, dt, steps)
    lv.device_status()
    got = lv.get_state().cpu().numpy()
    v = s0.cpu().numpy()
    del lv, s0
    torch.cuda.empty_cache()
    fab = orc.to_fab(v, 2)
    del v
    orc.rk4_advance(fab, 2, dx, orc.background(a_inv=2.0, c0=2.0, lambda_scale=2.0), 1.0, 0.0, dt, steps)
    ref = orc.from_fab(fab, 2)
    del fab
    assert _rel_max(got, ref) < 1e-12


@pytest.mark.parametrize("shape", [(64, 16, 40), (32, 8, 5), (96, 24, 70)])
def test_eval_rhs_f32_wide_staging_equals_cell_staging(axs, shape):
    """FP32 drop-in RHS: FABs with ng = 2 and tile-multiple extents stage their
    rows in 16-byte pieces, others cell by cell; same arithmetic, same bits."""
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + ny + nz)
    v = torch.from_numpy(rng.standard_normal((4, nz, ny, nx)) + 1.0).float().cuda()
    c = axs.Background.expanding(2.0, 2.0, lambda0=2.0).rhs_coeffs(1.7)
    out = []
    for ng in (2, 3):
        s = axs.new_fab((nx, ny, nz), ng, dtype=torch.float32)
        axs.valid(s, ng).copy_(v)
        axs.fill_periodic_ghosts(s, ng)
        r = axs.new_fab((nx, ny, nz), 0, dtype=torch.float32)
        axs.eval_rhs(s, r, ng, 0, 0.5, c)
        out.append(axs.valid(r, 0).clone())
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("kind", ["plain", "zeros", "wide", "edge28", "tiny", "large", "subnormal", "nonfinite"])
def test_f64_step_on_fields_of_every_exponent_range(axs, orc, kind):
    """One FP64 level step, whose Laplacians are summed as integers where every
    tap's exponent lies within 28 of the largest, against the stage-by-stage
    oracle: fields with exact zeros, exponents far apart, on both sides of the
    28, near the ends of the double range, and infinities and NaN (the same
    cells are finite). Tolerance: 1e-12 of the component's maximum, as for the
    other FP64 steps (13 taps of weight up to 30 in ulp of 2^-53, times
    h^2/dx^2 < 1)."""
    nx, ny, nz = shape = (24, 10, 9)
    rng = np.random.default_rng(11)
    v = rng.standard_normal((4, nz, ny, nx))
    if kind == "zeros":
        v[:, :, :, ::3] = 0.0
        v[3] = 0.0
    elif kind == "wide":
        v = np.ldexp(v, rng.integers(-70, 1, v.shape))
    elif kind == "edge28":
        v = np.ldexp(np.sign(v) * rng.uniform(1.0, 2.0, v.shape), -rng.integers(26, 31, v.shape) * (rng.random(v.shape) < 0.2))
    elif kind == "tiny":
        v *= 1e-160
    elif kind == "large":
        v *= 1e40
    elif kind == "subnormal":
        v *= 1e-308
    elif kind == "nonfinite":
        v[0, 2, 3, 4], v[1, 6, 7, 15], v[2, 4, 1, 20] = np.nan, np.inf, -np.inf
    dx, dt = 0.5, 0.05
    lam = 2.0 if kind != "large" else 1e-80
    bg, bgo = axs.Background.expanding(2.0, 1.0, lambda0=lam), orc.background(a_inv=2.0, c0=1.0, lambda_scale=lam)
    ref = orc.to_fab(v, 2)
    with np.errstate(all="ignore"):
        orc.rk4_advance(ref, 2, dx, bgo, 1.0, 0.0, dt, 1)
    ref = orc.from_fab(ref, 2)
    for cid, name in [(0, "default")] + axs.PeriodicLevel(shape, dx, dtype=torch.float64).tile_configs():
        lv = axs.PeriodicLevel(shape, dx, dtype=torch.float64, tile_config=cid)
        lv.set_state(_to_dev(v))
        lv.advance(bg, 1.0, 0.0, dt, 1)
        lv.device_status()
        got = lv.get_state().cpu().numpy()
        fin = np.isfinite(ref)
        np.testing.assert_array_equal(np.isfinite(got), fin, err_msg=name)
        for c in range(4):
            scale = max(np.abs(ref[c][fin[c]]).max(), 1e-307)
            assert np.abs(got[c] - ref[c])[fin[c]].max() <= 1e-12 * scale, (name, c)


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 1), (31, 5, 4), (33, 4, 9), (65, 3, 5), (127, 2, 3)])
@pytest.mark.parametrize("ng", [2, 3])
def test_f64_drop_in_kernels_on_rows_of_any_length(axs, orc, n, ng):
    """The FP64 RHS and the RK4 combination number the cells of the box through:
    rows shorter and longer than a warp, a box below a block, bit for bit."""
    nx, ny, nz = n
    rng = np.random.default_rng(sum(n) + ng)
    v = rng.standard_normal((4, nz + 2 * ng, ny + 2 * ng, nx + 2 * ng))
    soln = _to_dev(v)
    rhs = axs.new_fab(n, 1, dtype=torch.float64)
    axs.eval_rhs(soln, rhs, ng, 1, 0.3, axs._lib.RhsCoeffs(0.1, 1.3, 0.9))
    np.testing.assert_array_equal(axs.valid(rhs, 1).cpu().numpy(),
                                  orc.from_fab(orc.rhs(v, ng, 0.3, 0.1, 1.3, 0.9), ng))
    ks = [rng.standard_normal((4, nz, ny, nx)) * 10.0 ** rng.integers(-300, 300, (4, nz, ny, nx)) for _ in range(4)]
    ks[1][0], ks[2][1] = 0.0, 5e-324  # zeros and subnormals, which are doubled by another path
    ks[1][2, 0, 0, 0], ks[2][2, 0, 0, 0] = np.inf, 1.5e308
    u = rng.standard_normal((4, nz, ny, nx))
    d = axs.new_fab(n, ng, dtype=torch.float64)
    axs.rk4_combine(axs.valid(d, ng), _to_dev(u), *[_to_dev(k) for k in ks], 0, 0.6)
    with np.errstate(all="ignore"):
        ref = u + (0.6 / 6.0) * (((ks[0] + 2.0 * ks[1]) + 2.0 * ks[2]) + ks[3])
    np.testing.assert_array_equal(axs.valid(d, ng).cpu().numpy(), ref)


@pytest.mark.parametrize("ng", [2, 3])
def test_f32_rhs_of_part_of_a_box_equals_the_boxs(axs, ng):
    """The FP32 RHS marches 64 planes a block on a large box and down to 8 on a
    small one: the same bits for the same cells."""
    n = (256, 256, 192)
    g = torch.Generator(device="cuda").manual_seed(3)
    soln = axs.new_fab(n, ng, dtype=torch.float32)
    soln.normal_(generator=g)
    c = axs._lib.RhsCoeffs(0.1, 1.3, 0.9)
    big = axs.new_fab(n, 0, dtype=torch.float32)
    axs.eval_rhs(soln, big, ng, 0, 0.5, c)
    for (x, y, z), (nx, ny, nz) in [((0, 0, 0), (64, 64, 64)), ((32, 8, 5), (128, 128, 77)), ((3, 1, 7), (33, 17, 9)),
                                    ((64, 0, 100), (160, 200, 92)), ((1, 2, 3), (5, 4, 1))]:
        part = soln[:, z:z + nz + 2 * ng, y:y + ny + 2 * ng, x:x + nx + 2 * ng]
        out = axs.new_fab((nx, ny, nz), 1, dtype=torch.float32)
        axs.eval_rhs(part, out, ng, 1, 0.5, c)
        assert torch.equal(axs.valid(out, 1), big[:, z:z + nz, y:y + ny, x:x + nx]), (x, y, z, nx, ny, nz)


@pytest.mark.parametrize("dx", [0.5, 0.1, 0.3])
def test_f64_laplacian_weighs_no_site_alike_wrong(axs, dx):
    """What all sites' Laplacians have in common as an error: the slope of Pi's error after
    one step on its increment, against extended precision. dt = 3/128 makes h/6, h/3 and
    h^2/6 exact, so 1/(12 dx^2) is the one rounded weight; rounded to 53 bits and
    used as it is, it gives slopes of -5.6e-17, -3.1e-17 and -7.0e-17. Bound: 2^-56 =
    1.4e-17. (The rounding errors of 8192 values, 1.4e-16 of Pi at most each, give the
    slope an uncertainty of 2e-18 where increments are of Pi's size, which they exceed.)"""
    n, dt, ld = 16, 3.0 / 128.0, np.longdouble
    v = np.random.default_rng(8).standard_normal((4, n, n, n))
    v[2:] *= 0.2
    bg = axs.Background.expanding(2.0, 1.0, lambda0=2.0)
    lv = axs.PeriodicLevel(n, dx, dtype=torch.float64)
    lv.set_state(_to_dev(v))
    lv.advance(bg, 1.0, 0.0, dt, 1)
    lv.device_status()
    got = lv.get_state().cpu().numpy()

    def rhs(y, tau):
        c = bg.rhs_coeffs(tau)
        out = np.concatenate([y[2:], y[:2] * ld(c.kappa) - ld(c.lambda_) / 2 * ((y[:2] ** 2).sum(0) - ld(c.R2)) * y[:2]])
        lap = -90 * y[:2]
        for ax in (1, 2, 3):
            for k, w in ((1, 16), (2, -1)):
                lap = lap + w * (np.roll(y[:2], k, ax) + np.roll(y[:2], -k, ax))
        out[2:] += lap / (12 * ld(dx) * ld(dx))
        return out

    y, h = v.astype(ld), ld(dt)
    k1 = rhs(y, 1.0)
    k2 = rhs(y + h / 2 * k1, 1.0 + dt / 2)
    k3 = rhs(y + h / 2 * k2, 1.0 + dt / 2)
    ref = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + rhs(y + h * k3, 1.0 + dt))
    err, inc = (got - ref)[2:], (ref - y)[2:]
    assert abs(float((err * inc).sum() / (inc ** 2).sum())) < 2.0 ** -56


@pytest.mark.parametrize("shape", [(4, 2, 1), (16, 8, 2), (34, 9, 97), (98, 75, 50), (18, 130, 33), (130, 34, 7), (64, 64, 64)])
def test_f64_chunk_plans_cover_every_plane(axs, shape):
    """The FP64 sweeps' chunks of planes, planned by the fullest SM's work: levels of a
    few planes and of one chunk, uneven last chunks, more tiles than SMs and fewer. Every
    tiling has another plan and leaves the same bits, padding included; three steps."""
    nx, ny, nz = shape
    v = torch.from_numpy(np.random.default_rng(nx + ny + nz).standard_normal((4, nz, ny, nx))).cuda()
    v[:2] += 1.5
    bg = axs.Background.expanding(2.0, 1.0, lambda0=2.0)
    ref = None
    for cid, name in [(0, "default")] + axs.PeriodicLevel((16, 8, 2), 0.5, dtype=torch.float64).tile_configs():
        lv = axs.PeriodicLevel(shape, 0.5, dtype=torch.float64, tile_config=cid)
        lv.set_state(v)
        lv.advance(bg, 1.0, 0.0, 0.05, 3)
        lv.device_status()
        ref = lv.state.clone() if ref is None else ref
        assert torch.equal(lv.state, ref), name
