"""Several plasma species in the fused step.

A plasma split into two species of half the density each is the same plasma:
the charges and currents of the halves add up, and the force on an electron
does not depend on the species it is counted in.  The step with both halves
therefore gives the fields of the step with one species, up to the FP32
rounding of the deposits' sums.
"""
import numpy as np
import pytest
from conftest import BOX, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qp():
    import qpgpu

    return qpgpu


def step(qp, ind, densities, iter, graphs):
    c = qp.Context(ind[0], ind[1], ind[2], BOX)
    sp = [qp.Species2d(c, ppc=(2, 2), density=d) for d in densities]
    bm = qp.Beam3d(c, (16, 16, 32), gamma=20000.0, peak_density=2.0, center=(0.0, 0.0, 2.5),
                   sigma=(0.5, 0.5, 0.5))
    sim = qp.Simulation(c, sp, [bm], iter=iter, use_graphs=graphs)
    sim.step3d()
    out = dict(be=sim.get_3d("bexyz"), bb=sim.get_3d("bbxyz"), epw=sim.get_field("epw"),
               q3=sum(s.get_q3(c.nz // 2) for s in sp))
    for h in [sim, bm, *sp, c]:
        h.close()
    return out


@pytest.mark.parametrize("ind,iter,graphs", [((6, 6, 5), 1, False), ((6, 6, 5), 2, False),
                                             ((6, 5, 5), 3, True)])
def test_two_half_density_species_are_one_plasma(qp, ind, iter, graphs):
    one = step(qp, ind, [1.0], iter, graphs)
    two = step(qp, ind, [0.5, 0.5], iter, graphs)
    # FP32 sums of up to ~1e3 terms in another order (1e-6), carried through the
    # orbits of 32 slices: the run-to-run difference of one species is 1e-6 here
    assert rel_l2(two["be"], one["be"]) < 1e-4
    assert rel_l2(two["epw"], one["epw"]) < 1e-4
    assert rel_l2(two["q3"], one["q3"]) < 1e-4
    assert np.isfinite(two["bb"]).all()
