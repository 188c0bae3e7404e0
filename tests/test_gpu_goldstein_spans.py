"""Branch cuts gathered by several warps, and the fill's sweeps, at the sizes where the
spans, the residue list and the sweeps change form: maps shorter than a span's batch, sides
that no span divides, more residues than the list holds, a map without residues.  Charges
and cuts are whole numbers and match the oracle; the filled phase within 1e-4 rad RMSE."""
import numpy as np
import pytest

from test_gpu_goldstein import PHASE_TOL, noisy_phase, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,noise,least", [(4, 4, 2.0, 0), (5, 7, 2.0, 1), (61, 83, 1.0, 50), (83, 61, 1.0, 50),
                                             (129, 127, 0.0, 0), (200, 190, 3.0, 2049), (257, 255, 0.8, 50)])
def test_goldstein_spans(ctx, dev, oracle, w, h, noise, least):
    big = max(w, h)
    maps = np.stack([np.ascontiguousarray(noisy_phase(big, s, noise, 0.2)[:h, :w]) for s in (1, 2)])
    q, c, o, st = run_gpu(ctx, dev, maps)
    for a in range(len(maps)):
        oq = oracle.goldstein_residues(maps[a])
        assert np.array_equal(q[a], oq) and np.count_nonzero(oq) >= least
        oc = oracle.goldstein_cuts(oq)
        assert np.array_equal(c[a], oc)
        oo, ub, ost = oracle.goldstein_floodfill(oc, maps[a])
        assert st[a] == ost
        if ost == 0:
            assert np.sqrt(np.mean((o[a] - oo) ** 2)) < PHASE_TOL
