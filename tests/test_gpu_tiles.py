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
                                        (65, 1000, 31), (127, 257, 65), (96, 513, 100)])
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
