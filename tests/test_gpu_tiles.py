"""Line opacity at the sizes where the wavelength tiles and depth groups of the accumulation kernels end:
depth counts around a group, wavelength counts around a tile, few and many lines.

Tolerances.  FP64: each term carries a few ulps of the library functions (2e-16 each) and of the
evaluation, on the Gaussian flank 2 v^2 times those of v (v < 6 where a term matters): below 1e-13;
the bar is 1e-12 of LineOpac + ContOpac.  Mixed: FP32 terms and compensated sums, 2e-6 of LineOpac +
ContOpac (the path's bar)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def case(ntau, nwl, n, seed):
    from fastspec_b200 import workloads as W
    import fastspec_b200 as F
    st, cont = W.batch_atmosphere(5300.0, 4.2, ntau, {})
    step = 0.011
    grid = dict(wmode=0, wstart=5100.0, wend=5100.0 + (nwl - 0.5) * step, dstep=step)
    wave = F.make_grid(0, grid["wstart"], grid["wend"], step) + grid["wstart"]
    assert len(wave) == nwl
    lk = np.log(cont["cont_opac"])
    co = np.exp(np.stack([np.interp(wave, cont["cont_wave"], lk[:, t]) for t in range(ntau)], axis=1))
    L = W.atomic_lines(n, grid["wstart"], grid["wend"], seed, exact=False)
    return grid, st, co, L.arrays()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("ntau,nwl,n", [(3, 2, 1), (4, 63, 7), (5, 64, 9), (9, 65, 33), (31, 127, 40), (64, 129, 200),
                                        (65, 1000, 31), (127, 257, 65), (96, 513, 100), (8, 32, 16), (17, 33, 17)])
def test_tile_edges(fsg, oracle_mod, prec, ntau, nwl, n):
    grid, st, co, a = case(ntau, nwl, n, 17 * ntau + nwl)
    C = fsg.Context(precision=fsg.PREC_FP64 if prec == "fp64" else fsg.PREC_MIXED, vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    g = C.lineop_calc(fsg.LineList.from_arrays(a))
    S = oracle_mod.State(grid, st, contopac=co, vmicro=1.0)
    r = oracle_mod.lineop_calc(S, oracle_mod.Lines(**a, kind=2), list_type=2)
    np.testing.assert_array_equal(g["flags"] & 1, r["flags"] & 1)       # the mixed path marks no wide lines
    keep = (g["flags"] & 1) == 0
    np.testing.assert_array_equal(g["ileft"][keep], r["ileft"][keep])
    np.testing.assert_array_equal(g["iright"][keep], r["iright"][keep])
    err = np.max(np.abs(g["lineopac"] - r["lineopac"]) / (r["lineopac"] + co))
    assert err < (1e-12 if prec == "fp64" else 2e-6)
    C.close()


@pytest.mark.parametrize("step,nwl,n,eps", [(0.011, 300, 2500, 1e-10), (0.011, 4000, 9000, 1e-6), (9.0, 501, 4001, 1e-14)])
def test_paired_lines(fsg, step, nwl, n, eps):
    """Tiles with enough lines for the wing pass to take them two to a reciprocal: windows that cover all tiles,
    windows that end inside them, and (the last case) lines whose t^2 + 2a^2 leaves the range of a product, which
    stay single.  Mixed against FP64, the path's bar."""
    from fastspec_b200 import workloads as W
    ntau = 33
    _, st, _, _ = case(ntau, 2, 1, 0)
    w0 = 4000.0
    wave = fsg.make_grid(0, w0, w0 + (nwl - 0.5) * step, step) + w0
    co = np.tile(1e-2 * (1.0 + np.arange(ntau)), (len(wave), 1))
    L = fsg.LineList.from_arrays(W.atomic_lines(n, wave[0], wave[-1], nwl, exact=False).arrays())
    out = {}
    for prec in (fsg.PREC_FP64, fsg.PREC_MIXED):
        C = fsg.Context(precision=prec, vmicro=1.0, epsopac=eps)
        C.set_grid(0, w0, w0 + (nwl - 0.5) * step, step)
        C.set_atmosphere(st)
        C.set_contopac(co)
        out[prec] = C.lineop_calc(L)
        C.close()
    f, m = out[fsg.PREC_FP64], out[fsg.PREC_MIXED]
    keep = (f["flags"] & 1) == 0
    assert (f["iright"] - f["ileft"])[keep].astype(np.int64).sum() > 2048 * nwl     # lines to pair on a tile
    np.testing.assert_array_equal(f["ileft"][keep], m["ileft"][keep])
    assert np.max(np.abs(m["lineopac"] - f["lineopac"]) / (f["lineopac"] + co)) < 2e-6


@pytest.mark.parametrize("nwl,n", [(700, 40), (8001, 1500), (40001, 3000)])
def test_one_launch_equals_launch_per_class(fsg, nwl, n):
    """A list that fits one block takes its window-width classes in one launch, a longer one class by class (few and
    many depths a warp, whole groups of lines and remainders).  Sums of FP32 terms in another grouping: a rounding
    of 6e-8 for a class, 2e-7."""
    grid, st, co, a = case(33, nwl, n, 5)
    out = []
    for ram in (16.0, 0.75 * n * 1632e-9):               # the records of three quarters of the lines
        C = fsg.Context(vmicro=1.0, limitram_gb=ram)
        C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
        C.set_atmosphere(st)
        C.set_contopac(co)
        g = C.lineop_calc(fsg.LineList.from_arrays(a))
        out.append((g["stats"]["nblocks"], g["lineopac"]))
        C.close()
    assert out[0][0] == 1 and out[1][0] > 1
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=2e-7, atol=0.0)


@pytest.mark.parametrize("nwl,n", [(701, 60), (4001, 900), (24001, 10500)])
def test_class_sums_are_added_in_fp64(fsg, nwl, n):
    """Each window-width class is one compensated FP32 sum, and the classes are added in FP64, however long the list: a
    list in one launch for all classes equals the same list class by class (every class whole, in one block), to the
    rounding of some twenty FP64 additions.  Few enough lines on a tile that none are paired."""
    grid, st, co, a = case(33, nwl, n, 11)
    out = []
    for ram in (16.0, 0.8 * n * 1632e-9):                # all lines' records, or those of 80 % of them
        C = fsg.Context(vmicro=1.0, epsopac=3e-3, limitram_gb=ram)
        C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
        C.set_atmosphere(st)
        C.set_contopac(co)
        g = C.lineop_calc(fsg.LineList.from_arrays(a))
        out.append(g)
        C.close()
    keep = (g["flags"] & 1) == 0
    assert (n < 8192) == (np.count_nonzero(keep) <= 8192)
    width = (g["iright"] - g["ileft"] + 1)[keep]
    ncls = len(np.unique(np.ceil(np.log2(np.maximum(width, 256)))))
    assert out[0]["stats"]["nblocks"] == 1 and out[1]["stats"]["nblocks"] == ncls
    np.testing.assert_allclose(out[0]["lineopac"], out[1]["lineopac"], rtol=1e-14, atol=0.0)


@pytest.mark.parametrize("n", [32769, 45001])
def test_central_pass_forms(fsg, n):
    """Flags and windows do not depend on how the central pass spreads its lines: a list above 32,768 lines takes
    a thread per line, the parts of it a warp."""
    from fastspec_b200 import workloads as W
    grid, st, co, _ = case(31, 64, 1, 0)
    a = W.atomic_lines(n, grid["wstart"] - 40.0, grid["wend"] + 40.0, n, exact=False).arrays()

    def windows(a):
        C = fsg.Context(vmicro=1.0)
        C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
        C.set_atmosphere(st)
        C.set_contopac(co)
        g = C.lineop_calc(fsg.LineList.from_arrays(a))
        C.close()
        return np.stack([g["flags"], g["ileft"], g["iright"]])

    cut = [0, 300, 16000, n]
    parts = [windows({k: v[i:j] for k, v in a.items()}) for i, j in zip(cut, cut[1:])]
    np.testing.assert_array_equal(windows(a), np.concatenate(parts, axis=1))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("ntau,nwl,n", [(3, 2, 1), (4, 31, 5), (9, 33, 17), (33, 64, 20), (65, 300, 33), (128, 97, 12)])
def test_magnetic_tile_edges(fsg, oracle_mod, prec, ntau, nwl, n):
    """The same for Zeeman lines; errors on the scale of the depth's peak absorption profile (FP64: the
    offset of a component carries the rounding of lambda - lambda_c and of the shift, 2 v dv < 1e-13)."""
    from fastspec_b200 import workloads as W
    grid, st, co, _ = case(ntau, nwl, 1, 0)
    L = W.zeeman_lines(n, grid["wstart"], grid["wend"], 19 * ntau + nwl)
    z = W.zeeman_components(L, oracle_mod.zeeman_pattern)
    C = fsg.Context(precision=fsg.PREC_FP64 if prec == "fp64" else fsg.PREC_MIXED, vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    b = np.array([3000.0, 50.0, 20.0])
    g = C.mag_lineop_calc(fsg.LineList.from_arrays(L.arrays(), zeeman=z), 1, b)
    S = oracle_mod.State(grid, st, contopac=co, vmicro=1.0)
    r = oracle_mod.mag_lineop_calc(S, oracle_mod.Lines(**L.arrays(), kind=2, zeeman=z), 1, b)
    keep = (r["flags"] & 1) == 0
    np.testing.assert_array_equal((g["flags"] & 1) == 0, keep)
    np.testing.assert_array_equal(g["ileft"][keep], r["ileft"][keep])
    np.testing.assert_array_equal(g["iright"][keep], r["iright"][keep])
    om = r["maglineopac"]
    scale = np.maximum(om[..., :3].max(axis=(0, 2)), 1e-300)[None, :, None]
    assert np.max(np.abs(g["maglineopac"] - om) / scale) < (1e-12 if prec == "fp64" else 2e-6)
    C.close()


@pytest.mark.parametrize("prec,j", [("fp64", 5.0), ("fp64", 6.0), ("fp64", 17.0), ("mixed", 5.0), ("mixed", 6.0), ("mixed", 9.0)])
def test_many_zeeman_components(fsg, oracle_mod, prec, j):
    """Lines with more components than the tile kernel stages (32; a line J - J has 6 J, at J 17 the pi components
    alone are more).  Errors on the scale of the depth's peak absorption profile: FP64 as above; mixed, the FP32 sum of
    a profile's components, 6e-8 each, and ten operations a term."""
    from fastspec_b200 import workloads as W
    ntau, nwl, n = 33, 200, 12
    grid, st, co, _ = case(ntau, nwl, 1, 0)
    L = W.zeeman_lines(n, grid["wstart"], grid["wend"], int(j))
    few = L.zeeman
    L.zeeman = (np.where(np.arange(n) % 3 == 2, few[0], np.float32(j)), np.where(np.arange(n) % 3 == 2, few[1], np.float32(j)),
                few[2], few[3])
    z = W.zeeman_components(L, oracle_mod.zeeman_pattern)
    assert (z[0] + z[1]).max() == 6 * j
    C = fsg.Context(precision=fsg.PREC_FP64 if prec == "fp64" else fsg.PREC_MIXED, vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    b = np.array([3000.0, 50.0, 20.0])
    g = C.mag_lineop_calc(fsg.LineList.from_arrays(L.arrays(), zeeman=z), 1, b)
    S = oracle_mod.State(grid, st, contopac=co, vmicro=1.0)
    r = oracle_mod.mag_lineop_calc(S, oracle_mod.Lines(**L.arrays(), kind=2, zeeman=z), 1, b)
    om = r["maglineopac"]
    scale = np.maximum(om[..., :3].max(axis=(0, 2)), 1e-300)[None, :, None]
    tol = 1e-12 if prec == "fp64" else 6e-8 * (10 + 2 * j + 1)
    assert np.max(np.abs(g["maglineopac"] - om) / scale) < tol
    C.close()


@pytest.mark.parametrize("ntau,nwl,nmu", [(3, 2, 1), (4, 7, 2), (64, 9, 9), (65, 17, 16), (128, 8, 5)])
def test_solver_edges(fsg, oracle_mod, ntau, nwl, nmu):
    """The formal solver around its CTA's eight wavelengths and its thread counts, on a line opacity spread over
    nine decades of the continuum's.  Bar: 1e-10 relative, as for the drivers (the DELO differences amplify a
    rounding of the exponential 1e7 times just above the Taylor branch)."""
    grid, st, co, _ = case(ntau, nwl, 1, 0)
    lo = co * 10.0 ** np.random.default_rng(ntau + nwl).uniform(-4.0, 5.0, co.shape)
    x, w, _ = fsg.mu_quadrature(1, nmu)
    C = fsg.Context(vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    C.set_mu(x, w)
    C.lineop_set(lo)
    spl, spc, sfl, sfc = C.radtran()
    S = oracle_mod.State(grid, st, contopac=co, vmicro=1.0)
    ospl, ospc = oracle_mod.radtran(S, x, lo)
    osfl, osfc = oracle_mod.disk_integ(w, ospl, ospc)
    for a, b in ((spl, ospl), (spc, ospc), (sfl, osfl), (sfc, osfc)):
        assert np.max(np.abs(a / b - 1)) < 1e-10
    C.close()


def test_central_pass_forms_shallow(fsg):
    """The same in a shallow model, where shorter lists take a thread per line (8 depths: above 7,600)."""
    from fastspec_b200 import workloads as W
    grid, st, co, _ = case(8, 64, 1, 0)
    a = W.atomic_lines(9001, grid["wstart"] - 40.0, grid["wend"] + 40.0, 2, exact=False).arrays()
    C = fsg.Context(vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    out = [C.lineop_calc(fsg.LineList.from_arrays({k: v[i:j] for k, v in a.items()})) for i, j in ((0, 9001), (0, 5000), (5000, 9001))]
    for k in ("flags", "ileft", "iright"):
        np.testing.assert_array_equal(out[0][k], np.concatenate([out[1][k], out[2][k]]))
    C.close()


@pytest.mark.parametrize("sphere", [False, True])
def test_solver_without_opacity(fsg, oracle_mod, sphere):
    """Layers whose opacities cancel to 0, are infinite or are no number: optical-depth steps of 0, whose reciprocals
    are infinite.  The intensities are numbers exactly where the oracle's are; those within 1e-10 of the disk-centre
    continuum, the bar of the intensities."""
    ntau, nwl, nmu = 56, 160, 5
    grid, st, co, _ = case(ntau, nwl, 1, 0)
    x, w, _ = fsg.mu_quadrature(1, nmu)
    lo = co * 10.0 ** np.random.default_rng(7).uniform(-2.0, 2.0, co.shape)
    k = 0
    for run in (1, 2, 3, 6):
        for d in (0, 1, 7, 20, 21, 22, ntau - run - 1, ntau - run):
            lo[k, d:d + run] = -co[k, d:d + run]
            k += 1
    for v in (np.inf, -np.inf, np.nan):
        for d in (0, 1, 25, ntau - 2, ntau - 1):
            lo[k, d] = v
            k += 1
    assert k < nwl
    C = fsg.Context(vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    C.set_mu(x, w)
    S = oracle_mod.State(grid, st, contopac=co, vmicro=1.0)
    if sphere:
        from fastspec_b200 import workloads as W
        h = W.model_heights(st["rhox"], st["rho"])
        radius = 250.0 * float(h[0] - h[-1])
        C.set_geometry(radius, h)
        S.set_sphere(radius, h, x)
    C.lineop_set(lo)
    spl, spc, _, _ = C.radtran()
    ospl, ospc = oracle_mod.radtran(S, x, lo)
    np.testing.assert_array_equal(np.isfinite(spl), np.isfinite(ospl))
    ok = np.isfinite(ospl)
    assert 0 < np.count_nonzero(~ok) < ok.size // 2
    assert np.max((np.abs(spl - ospl) / ospc[:, :1])[ok]) < 1e-10
    C.close()


@pytest.mark.parametrize("nwl,nmu,vsini,vmacro,vgau", [(9, 2, 0.0, 0.0, 0.0), (9, 3, 30.0, 5.0, 2.0e4), (640, 7, 12.0, 0.0, 0.0),
                                                       (641, 16, 0.0, 3.0, 9.0e4), (1283, 5, 40.0, 6.0, 5.0),
                                                       (3000, 1, 7.0, 2.0, 0.0), (14001, 3, 900.0, 90.0, 3.0e3)])
def test_broadening_edges(fsg, oracle_mod, nwl, nmu, vsini, vmacro, vgau):
    """The broadened flux around the tile of 640 wavelengths, with kernels wider than the spectrum and (the last
    case: 6,000 points either side) wider than the staged halo allows.  Sums of positive products: 1e-16 each,
    12,000 of them at most, below 1e-12."""
    import torch
    R = 2.0e6 if vsini > 100.0 else 3.0e5
    dstep = 2.99792458e5 / R
    grid = dict(wmode=1, wstart=5000.0, wend=5000.0 * np.exp((nwl - 0.5) / R), dstep=dstep)
    x, w, r = fsg.mu_quadrature(1, nmu)
    C = fsg.Context()
    wave = C.set_grid(1, grid["wstart"], grid["wend"], dstep) + grid["wstart"]
    assert len(wave) == nwl
    C.set_mu(x, w)
    rng = np.random.default_rng(nwl)
    spc = rng.uniform(0.9, 1.1, (nwl, nmu))
    spl = spc * rng.uniform(0.05, 1.0, (nwl, nmu))
    d = [torch.from_numpy(a).cuda() for a in (spl, spc)] + [torch.empty(nwl, dtype=torch.float64, device="cuda")
                                                            for _ in range(2)]
    torch.cuda.synchronize()
    C.disk_integ_conv_dev(r, vsini, vmacro, vgau, *[t.data_ptr() for t in d])
    osfl, osfc = oracle_mod.disk_integ_conv(x, w, r, spl, spc, oracle_mod.grid_dv(grid, wave), vsini, vmacro,
                                            oracle_mod.gauss_sigma_pix(grid, wave, vgau) if vgau > 0 else 0.0)
    assert np.max(np.abs(d[2].cpu().numpy() / osfl - 1)) < 1e-12
    assert np.max(np.abs(d[3].cpu().numpy() / osfc - 1)) < 1e-12
    C.close()


@pytest.mark.parametrize("ntau,nwl", [(9, 31000), (56, 6001), (64, 4801)])
def test_adjoint_forms_agree(fsg, ntau, nwl):
    """The adjoint's line pass takes fewer points a warp where there are few tiles: the gradients of ranges short enough
    for that, summed, against the whole grid's.  FP32 profiles summed in other groups, both signs: 2e-6 of the sum of
    magnitudes, as at the tile edges."""
    import torch
    from fastspec_b200.shard import GpuBackend
    grid, st, co, a = case(ntau, nwl, 150, 13)
    C = fsg.Context(vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    x, w, _ = fsg.mu_quadrature(1, 2)
    C.set_mu(x, w)
    B = GpuBackend(fsg, C, {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in a.items()})
    C.lineop_reset()
    C.lineop_calc_dev(B.full)
    win = B.central(0, B.n, B.n)
    g = torch.from_numpy(np.random.default_rng(3).normal(0.0, 1.0, nwl)).cuda()
    whole = B.adjoint(win, 1, nwl, g)
    warps = lambda n: ((n - 1) // 128 + 1) * ((ntau + 3) // 4)       # noqa: E731
    cut = nwl // 3
    ranges = ((1, cut), (cut + 1, 2 * cut + 5), (2 * cut + 6, nwl))
    assert warps(nwl) >= 600 and all(warps(j - i + 1) < 600 for i, j in ranges)
    parts = [B.adjoint(win, i, j, g) for i, j in ranges]
    for q in range(2):
        total = sum(p[q] for p in parts)
        assert float((total - whole[q]).abs().max()) < 2e-6 * float(whole[q].abs().sum())
    C.close()


@pytest.mark.parametrize("ntau,nwl,n", [(3, 2, 1), (7, 127, 8), (9, 129, 9), (33, 300, 33), (65, 640, 70)])
def test_adjoint_tile_edges(fsg, ntau, nwl, n):
    """The line pass of the adjoint around its tiles and depth groups: the whole-grid gradients against the sum of
    those of two ranges (split inside a tile), and, where every window covers the grid, dL/d ln gf of the whole
    list, which then is the sum of dL/dkappa * LineOpac, against that sum on the FP64 opacity.  The profiles are FP32 (6e-8 per
    operation, some ten of them, summed with both signs): 2e-6 of the sum of magnitudes."""
    import ctypes
    import torch
    from fastspec_b200.shard import GpuBackend
    grid, st, co, a = case(ntau, nwl, n, 5 * ntau + nwl)
    C = fsg.Context(precision=fsg.PREC_FP64, vmicro=1.0, epsopac=1e-12)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    x, w, _ = fsg.mu_quadrature(1, 3)
    C.set_mu(x, w)
    dt = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in a.items()}
    B = GpuBackend(fsg, C, dt)
    e = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")      # noqa: E731
    sfl, sfc, gk = e(nwl), e(nwl), e(nwl, ntau)
    win = torch.zeros((3, n), dtype=torch.int32, device="cuda")
    C.lineop_reset()
    C.lineop_calc_dev(B.full)
    C.radtran_dev(None, None, sfl.data_ptr(), sfc.data_ptr())
    C.central_dev(B.full, win[0].data_ptr(), win[1].data_ptr(), win[2].data_ptr())
    keep = (win[0] & 1) == 0
    covered = bool(((win[1] == 1) & (win[2] == nwl))[keep].all())            # no window edge moves with gf
    gf = torch.from_numpy(np.random.default_rng(n).normal(0.0, 1.0, nwl)).cuda() / sfc
    out = [(e(n), e(n)) for _ in range(3)]
    torch.cuda.synchronize()
    C.adjoint_dev(B.full, gf.data_ptr(), out[0][0].data_ptr(), out[0][1].data_ptr(), gk.data_ptr())
    cut = nwl // 2
    for (i0, i1), o in zip(((1, cut), (cut + 1, nwl)), out[1:]):
        C.adjoint_range_dev(B.full, win[0].data_ptr(), win[1].data_ptr(), win[2].data_ptr(), i0, i1, gf.data_ptr(),
                            o[0].data_ptr(), o[1].data_ptr())
    lo = torch.from_numpy(C.lineop_get()).cuda()
    scale = float((gk * lo).abs().sum())
    if covered:
        assert abs(float(out[0][0].sum()) - float((gk * lo).sum())) < 2e-6 * scale
    for q in range(2):
        assert float((out[0][q] - out[1][q] - out[2][q]).abs().max()) < 2e-6 * max(scale, float(out[0][q].abs().sum()))
    C.close()


@pytest.mark.parametrize("ntau,nwl", [(5, 3000), (56, 7501), (71, 8001)])
def test_fp64_forms_sum_alike(fsg, ntau, nwl):
    """The FP64 tile kernel takes fewer points a warp where there are few wavelengths: ranges short enough for each of
    its forms give the sums of the whole grid bit for bit."""
    import torch
    from fastspec_b200.shard import GpuBackend
    grid, st, co, a = case(ntau, nwl, 300, 9)
    C = fsg.Context(precision=fsg.PREC_FP64, vmicro=1.0)
    C.set_grid(grid["wmode"], grid["wstart"], grid["wend"], grid["dstep"])
    C.set_atmosphere(st)
    C.set_contopac(co)
    B = GpuBackend(fsg, C, {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in a.items()})
    C.lineop_reset()
    C.lineop_calc_dev(B.full)
    whole = C.lineop_get()
    win = B.central(0, B.n, B.n)
    warps = lambda n: ((n - 1) // 64 + 1) * ((ntau + 3) // 4)        # noqa: E731
    used = set()
    for i0, i1 in ((1, 1), (17, 80), (33, 1003), (100, 2999), (60, min(5500, nwl)), (1, nwl)):
        used.add((warps(i1 - i0 + 1) >= 660) + (warps(i1 - i0 + 1) >= 1600))
        B.accumulate(win, i0, i1)
        assert np.array_equal(C.lineop_get()[i0 - 1:i1], whole[i0 - 1:i1])
    assert len(used) == (1 if ntau == 5 else 3)
    C.close()
