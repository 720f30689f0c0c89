"""The grid kernels against numpy at axis lengths with every kind of factor (4, 2, 3, 5, other primes,
1) and odd and even halves.  Tolerances: FP64 transforms of N points err by a few u log2 N relative to
the largest value (u = 1.1e-16); 1e-13 leaves a factor of 50."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 8), (7, 12, 15), (9, 10, 11), (25, 6, 13), (16, 27, 5), (14, 22, 17), (45, 32, 30), (12, 9, 2),
          (36, 64, 75)]


def _ops(shape, natoms=3):
    from lresdft_gb300 import LResGPU, system
    from lresdft_gb300.scf import GridOps
    rng = np.random.default_rng(sum(shape))
    cell = 0.5 * np.array(shape, float)
    pos = rng.uniform(0, 1, (natoms, 3)) * cell
    cr = system.Crystal(pos, np.ones(natoms), cell, shape, 1.0, rcs=rng.uniform(0.3, 0.8, natoms))
    b = system.LCAOBasis(cr, rcut=min(0.9, 0.45 * cell.min()), s_exps=(1.0,), p_exps=())
    s = LResGPU(b, cr.pos[:1], R_w=1e3, M=2, precision="mixed", route="ldl", trace_rows=False)
    return cr, s, GridOps(s)


@pytest.mark.parametrize("shape", SHAPES)
def test_hartree_and_ion(shape):
    cr, s, go = _ops(shape)
    rng = np.random.default_rng(1)
    dens = rng.uniform(0, 1, shape) ** 4
    k = [2 * np.pi * np.fft.fftfreq(m, L / m) for m, L in zip(shape, cr.cell)]
    K = np.meshgrid(*k, indexing="ij")
    g2 = sum(x * x for x in K)
    g2[0, 0, 0] = np.inf
    want = np.real(np.fft.ifftn(4 * np.pi * np.fft.fftn(dens) / g2))
    got = go.lda_hartree(dens)[2]
    assert np.max(np.abs(got - want)) <= 1e-13 * np.max(np.abs(want))
    vg = np.zeros(shape, complex)
    for R, z, rc in zip(cr.pos, cr.Z, cr.atom_rc):
        vg += z * np.exp(-1j * sum(x * r for x, r in zip(K, R)) - np.where(np.isinf(g2), 0, g2) * rc * rc / 4)
    want = np.real(np.fft.ifftn(-4 * np.pi * vg / g2 / np.prod(cr.cell))) * cr.ng
    got = go.ion_potential()
    # (the phases K.R of the corner of the spectrum are ~100, rounded to 1e-14)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    s.close()


def test_lda_range():
    """Densities from below the floor through both branches (rs = 1 at n = 3 / (4 pi)) to huge values,
    inf and NaN as the formula treats them.  A handful of rounded operations per value: 4e-15."""
    cr, s, go = _ops((8, 9, 10))
    n = np.geomspace(1e-18, 1e40, cr.ng)
    n[:6] = [0.0, -1.0, 1e-14, 3 / (4 * np.pi), np.nextafter(3 / (4 * np.pi), 1), np.nextafter(3 / (4 * np.pi), 0)]
    nn = np.maximum(n, 1e-14)
    rs = (3 / (4 * np.pi * nn)) ** (1 / 3)
    ex = -0.75 * (3 * nn / np.pi) ** (1 / 3)
    sr, lr = np.sqrt(rs), np.log(rs)
    den = 1 + 1.0529 * sr + 0.3334 * rs
    ec = np.where(rs >= 1, -0.1423 / den, 0.0311 * lr - 0.048 + 0.002 * rs * lr - 0.0116 * rs)
    vc = np.where(rs >= 1, -0.1423 / den * (1 + 7 / 6 * 1.0529 * sr + 4 / 3 * 0.3334 * rs) / den,
                  0.0311 * lr - 0.048 - 0.0311 / 3 + 2 / 3 * 0.002 * rs * lr + (-0.0232 - 0.002) / 3 * rs)
    exc, vxc, _ = go.lda_hartree(n.reshape(cr.shape))
    # (the two branches meet with a jump of 3e-5 at rs = 1: those three points are compared loosely)
    tol = np.full(cr.ng, 4e-15)
    tol[3:6] = 1e-4
    assert np.all(np.abs(exc.ravel() - (ex + ec)) <= tol * np.abs(ex + ec))
    assert np.all(np.abs(vxc.ravel() - (4 / 3 * ex + vc)) <= tol * np.abs(4 / 3 * ex + vc))
    n[:] = 0.1
    n[:3] = [np.inf, np.nan, 1e308]
    exc, _, _ = go.lda_hartree(n.reshape(cr.shape))
    e = exc.ravel()
    assert not np.isfinite(e[0]) and np.isfinite(e[2])
    assert e[1] == pytest.approx(-0.75 * (3 * 1e-14 / np.pi) ** (1 / 3) - 0.1423 / (1 + 1.0529 * (3 / (4e-14 * np.pi)) ** (1 / 6) + 0.3334 * (3 / (4e-14 * np.pi)) ** (1 / 3)))
    s.close()
