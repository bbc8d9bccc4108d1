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


# the x passes of their cbq ride along up to 4 species and stand alone beyond;
# more than 8 need launches of their own to clear their currents and sum their
# charges in two parts (16 planes each), more than 12 smooth in two launches
@pytest.mark.parametrize("n", [4, 5, 8, 9, 13])
def test_many_species_are_one_plasma(qp, n):
    one = step(qp, (6, 5, 4), [1.0], 2, False)
    many = step(qp, (6, 5, 4), [1.0 / n] * n, 2, n % 2 == 1)
    for name in ("be", "bb", "epw", "q3"):  # the bar as above
        assert rel_l2(many[name], one[name]) < 1e-4, name


@pytest.mark.parametrize("nspecies", [1, 3])
def test_particles_restored_between_slices_give_the_same_slices(qp, nspecies):
    """A caller that puts a species' particles back between two slices (here the
    ones it has just read, in another order) gets the slices it would have got
    without: the charge of the next slice is formed from what it put there."""
    def run(restore):
        c = qp.Context(6, 6, 5, BOX)
        sp = [qp.Species2d(c, ppc=(2, 2), density=1.0 / nspecies) for _ in range(nspecies)]
        bm = qp.Beam3d(c, (16, 16, 32), gamma=20000.0, peak_density=2.0, center=(0.0, 0.0, 2.5),
                       sigma=(0.5, 0.5, 0.5))
        sim = qp.Simulation(c, sp, [bm], iter=1)
        sim.begin3d()
        sim.slices(15)
        if restore:
            for s in sp:
                pp, kp = s.get_particles()
                pp[7] *= 0.5  # wrong charges, which must be gone again below
                s.set_particles(pp, kp)
                pp[7] *= 2.0
                for t in range(s.ntiles):
                    pp[:, : kp[t], t] = pp[:, : kp[t], t][:, ::-1]
                s.set_particles(pp, kp)
        sim.slices(17)
        sim.end3d()
        be = sim.get_3d("bexyz")
        for h in [sim, bm, *sp, c]:
            h.close()
        return be

    assert rel_l2(run(True), run(False)) < 1e-5  # FP32 sums in another order


@pytest.mark.parametrize("ind", [(4, 4), (6, 5), (5, 9)])
def test_field_algebra_runs_components_in_the_lists_order(qp, ind):
    """mult / add / sub over component lists, several of them in one launch: the
    same as one component after another, also where a component reads what an
    earlier one of the list wrote, and for planes that do not fill a launch's CTAs
    evenly."""
    c = qp.Context(ind[0], ind[1], 1, BOX)
    rng = np.random.default_rng(3)
    a, b = qp.Field2d(c, 3), qp.Field2d(c, 3)
    va, vb = (rng.standard_normal(c.ks_shape(3)).astype(np.float32) for _ in range(2))
    cases = [("mult", a, None, [1, 2], [2, 1], [2.0, 3.0]), ("mult", b, None, [1, 3], [3, 1], [0.5, -1.0]),
             ("add", a, b, [1, 2, 3], [2, 1, 3], [1, 3, 2]), ("sub", a, b, [2, 1], [1, 2], [2, 2])]
    for op, x, y, d, d1, third in cases:
        a.set_ks(va)
        b.set_ks(vb)
        ref = {id(a): va.copy(), id(b): vb.copy()}
        for i in range(len(d)):
            src = ref[id(x)][d1[i] - 1]
            if op == "mult":
                ref[id(a)][d[i] - 1] = src * np.float32(third[i])
            else:
                o = ref[id(y)][third[i] - 1]
                ref[id(a)][d[i] - 1] = src + o if op == "add" else src - o
        if op == "mult":
            a.mult(x, third, dim=d, dim1=d1)
        else:
            getattr(a, op)(x, y, dim=d, dim1=d1, dim2=third)
        assert np.array_equal(a.get_ks(), ref[id(a)])
    for h in (a, b, c):
        h.close()


def test_charge_between_slices_is_the_last_slices(qp):
    """Between slices() calls get_q() of one of several species is the charge
    that the last slice ran with, that of the particles as they were before it,
    after an odd and after an even number of slices."""
    def run(chunks):
        c = qp.Context(6, 5, 4, BOX)
        sp = [qp.Species2d(c, ppc=(2, 2), density=d) for d in (0.75, 0.25)]
        bm = qp.Beam3d(c, (16, 16, 32), peak_density=2.0, center=(0.0, 0.0, 2.5),
                       sigma=(0.5, 0.5, 0.5))
        sim = qp.Simulation(c, sp, [bm], iter=1)
        sim.begin3d()
        assert not any(s.get_q().any() for s in sp)
        seen, done = {}, 0
        for n in chunks:
            before = [s.get_particles() for s in sp]
            sim.slices(n)
            done += n
            seen[done] = (before, [s.get_q() for s in sp])
        sim.end3d()
        be = sim.get_3d("bexyz")
        for h in (sim, bm, *sp, c):
            h.close()
        return seen, be

    single, be1 = run([1] * 16)
    several, be2 = run([2, 3, 1, 4, 1, 1, 4])
    assert rel_l2(be2, be1) < 1e-5
    c2 = qp.Context(6, 5, 4, BOX)
    s2, qe = qp.Species2d(c2, ppc=(2, 2)), qp.Field2d(c2, 1)
    for j in several:
        for k in range(2):
            pp, kp = single[j][0][k]
            s2.set_particles(pp, kp)
            qe.as_(0.0)
            s2.qdp(qe)
            want = s2.get_q()
            assert rel_l2(single[j][1][k], want) < 1e-6  # FP32 sums in another order
            assert rel_l2(several[j][1][k], want) < 1e-5  # of another run
    for h in (s2, qe, c2):
        h.close()
