"""Kernels whose launch shape follows the batch: the same system gives the
same forces and energies whatever shares the batch with it, and the shapes'
edges (few and many members, partial groups) match the oracle."""
import numpy as np
import pytest

from q_b200 import FP64, MIXED, Batch, System, synth
from tests.oracle_binding import load_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-11), (MIXED, 1e-11)])
@pytest.mark.parametrize("nq", [3, 20])
def test_q_water_warps_per_group(tmp_path, precision, tol, nq):
    """k_nb_qw with 8, 4 and 1 warps per water group (1, 50 and 170 systems),
    fewer Q atoms than warps and more than a staging chunk.  The FP32 sums do
    not depend on the shape, so both engines agree to FP64 rounding: sums of
    ~1e3 terms, 1e3 x 2^-53 = 1e-13 of the largest, bar 1e-11."""
    base = synth.fep_solute(str(tmp_path), radius=12.0, seed=5)
    g = synth.perturbation(base, "p%d" % nq, list(range(nq)), 0.2, 0.6, seed=5)
    systems = [System.open(g.inp, lambdas=(0.4, 0.6), seed=3) for _ in range(170)]
    ref = None
    for n in (1, 50, 170):
        b = Batch(systems[:n], precision=precision)
        b.set_tuning(lrf_tiles_per_block=1)      # the LRF's FP32 partial sums follow it
        b.evaluate(precision == FP64)
        grad, (E, EQ) = b.gradient(n - 1), b.energy_vectors(n - 1)
        if ref is None:
            ref = (grad, EQ)
        scale = np.abs(ref[0]).max()
        assert np.abs(grad - ref[0]).max() <= tol * scale, n
        assert np.abs(EQ - ref[1]).max() <= tol * max(1.0, np.abs(ref[1]).max()), n
        b.close()


@pytest.mark.parametrize("radius", [5.0, 9.0, 27.0])
def test_polarisation_shells_match_oracle(tmp_path, radius):
    """k_watpol at shells of a few members and of more than a block's threads:
    the restraint's energy and the whole gradient against the oracle (the
    repository's bar: 1e-3 kcal/mol, gradients 1e-4 relative)."""
    g = synth.water_sphere(str(tmp_path), radius=radius, seed=77)
    s = System.open(g.inp, seed=5)
    b = Batch([s], precision=FP64)
    b.evaluate(True)
    o = load_oracle().create(s)
    o.final_energy()
    assert np.abs(b.energy_vectors(0)[0] - o.energy_vectors()[0]).max() < 1e-3
    go = o.gradient()
    assert np.abs(b.gradient(0) - go).max() < 1e-4 * np.abs(go).max()
