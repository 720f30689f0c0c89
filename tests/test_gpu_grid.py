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
