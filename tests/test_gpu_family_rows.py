"""The family pass takes a warp or a thread per row by the number of rows.  On both
sides of every limit (152 SMs): idist, fac and the surface factors fncst against
numpy doing the same operations, the sums in the order of a warp's tree, bit for
bit; w and m to 1e-13 (another exp)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(dims, dx):
    grids = np.meshgrid(*[np.arange(n) - n / 2.0 + 0.5 for n in dims], indexing="ij")
    return [g.ravel(order="F") * dx for g in grids]


def _bonds(eng):
    rowptr, nl = eng.csr()
    n = np.diff(rowptr)
    row = np.repeat(np.arange(len(n)), n)
    return row, nl, np.arange(len(nl)) - rowptr[row], len(n)


def _tree(values, row, place, rows):
    """Sum per row: lane place % 32 adds its values in order, then the lanes in
    halves (16, 8, 4, 2, 1)."""
    acc = np.zeros((rows, 32))
    for turn in range(int(place.max()) // 32 + 1):
        at = place // 32 == turn
        acc[row[at], place[at] % 32] += values[at]
    for off in (16, 8, 4, 2, 1):
        acc = acc[:, :off] + acc[:, off:2 * off]
    return acc[:, 0]


def _check(p, coords, energies, weights):
    from pd_gpu1_gb300.engine import Engine

    dim = p.dim
    with Engine(p) as eng:
        eng.set_coords(*coords)
        eng.find_neighbor_gpu()
        if energies:
            eng.surface_correct_gpu()
        elif weights:
            eng.initial_weight()
        else:
            eng.vol_corr()
        got = {f: eng.get(f) for f in ("IDIST", "FAC") + (("FNCST_X", "FNCST_Y", "FNCST_Z") if energies else ()) +
               (("W", "M") if weights else ())}
        row, nl, place, rows = _bonds(eng)
    c, i = [a[nl] for a in coords], [a[row] for a in coords]
    sq = [(a - b) * (a - b) for a, b in zip(c, i)]
    L0 = np.sqrt(sq[0] + sq[1] if dim == 2 else sq[0] + sq[1] + sq[2])
    inner, outer = p.delta - p.dx / 2.0, p.delta + p.dx / 2.0
    f = np.where(L0 <= inner, 1.0, np.where(L0 <= outer, (outer - L0) / p.dx, 0.0))
    np.testing.assert_array_equal(got["IDIST"], L0)
    np.testing.assert_array_equal(got["FAC"], f)
    if energies:
        sed = 0.6 * p.emod * 1.0e-6 if dim == 3 else 0.5 * p.emod / (1.0 - p.pratio * p.pratio) * 1.0e-6
        for a in range(dim):
            dd = c[a] + 0.001 * c[a] - i[a] - 0.001 * i[a]
            e = list(sq)
            e[a] = dd * dd
            L = np.sqrt(e[0] + e[1] if dim == 2 else e[0] + e[1] + e[2])
            t = 0.25 * p.bc * (L - L0) * (L - L0) / L0 * p.vol * f
            with np.errstate(divide="ignore"):  # a single row of nodes has no energy across it
                want = sed / _tree(t, row, place, rows)
            np.testing.assert_array_equal(got["FNCST_" + "XYZ"[a]], want)
    if weights:
        w = np.exp(-(L0 * L0) / (p.delta * p.delta))
        np.testing.assert_allclose(got["W"], w, rtol=1e-13)
        np.testing.assert_allclose(got["M"], _tree(w * (L0 * L0) * p.vol * f, row, place, rows), rtol=1e-13)


def _params(dim, model, dims, dx):
    from pd_gpu1_gb300.engine import derive_params

    p = derive_params(dim, model, 2, 1e-7, 1, dx, 0.0, dx, 0.01, 0.01, 0.01, 192e9, 0.25, 8000.0, 0.04472)
    p.N = p.N_int = int(np.prod(dims))
    p.MN = 32 if dim == 2 else 128
    return p


# few rows, and 80 and 168 rows an SM: 12,160 and 25,536
@pytest.mark.parametrize("energies", [False, True])
@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("dims", [(2, 3), (16, 1), (31, 33), (110, 110), (111, 110), (160, 159), (160, 160)])
def test_plates(dims, model, energies):
    dx = 1e-4
    _check(_params(2, model, dims, dx), _lattice(dims, dx), energies, model == 2)


# 188, 190, 310, 420 and 470 rows an SM: 28,576, 28,880, 47,120, 63,840 and 71,440
@pytest.mark.parametrize("model,energies", [(1, False), (1, True), (2, False), (2, True)])
@pytest.mark.parametrize("dims", [(2, 2, 2), (9, 8, 7), (56, 56, 9), (57, 56, 9), (57, 57, 9), (72, 72, 9), (73, 72, 9), (84, 84, 9),
                                  (85, 84, 9), (89, 89, 9), (90, 89, 9)])
def test_blocks(dims, model, energies):
    dx = 1e-3
    _check(_params(3, model, dims, dx), _lattice(dims, dx), energies, model == 2)
