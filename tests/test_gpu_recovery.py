"""A tile or inbox that overflows inside the fused step: the host grows the
buffers, redoes the push, stores and charge of that slice and goes on, and the
slices after it (all of them enqueued before the host looks) have left the
state alone.  A plasma that is set to converge on one tile (momentum -a r: its
density grows to (1 - a)^-2 within a quarter of a plasma wavelength) overflows
buffers made for little more than the loaded density; the same step with room
from the start is the reference.  The two runs differ by the order of FP32
sums: 1e-6 per slice, carried through 32 slices; the bar is that of the
whole-step tests."""
import numpy as np
import pytest
from conftest import BOX, rel_l2

FINE = [[-3.0, 3.0], [-3.0, 3.0], [0.0, 10.0]]  # tiles of 0.75 c/wp: a mild density peak fills one

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qp():
    import qpgpu

    return qpgpu


def converge(sp, a=0.4):
    pp, kp = sp.get_particles()
    live = np.arange(pp.shape[1])[:, None] < kp[None, :]
    dx, dy = pp[0] - 56.0, pp[1] - 56.0  # the centre of a tile
    inside = live & (dx * dx + dy * dy < 20.0 ** 2)
    pp[2] -= np.where(inside, a * dx, 0).astype(np.float32)
    pp[3] -= np.where(inside, a * dy, 0).astype(np.float32)
    sp.set_particles(pp, kp)


def step(qp, xtras, nspecies=1, graphs=False, predict=0, record=False):
    c = qp.Context(7, 7, 5, FINE)
    sp = [qp.Species2d(c, ppc=(2, 2), density=1.0 / nspecies, xtras=xtras)
          for _ in range(nspecies)]
    bm = qp.Beam3d(c, (32, 32, 32), peak_density=1.0, center=(0.0, 0.0, 2.5),
                   sigma=(0.5, 0.5, 0.5))
    sim = qp.Simulation(c, sp, [bm], iter=2, use_graphs=graphs, predict=predict)
    extra = []
    if predict == 3:
        extra.append(qp.Predictor(seed=1))  # untrained: the quadratic extrapolation
        sim.set_predictor(extra[0])
    data = qp.TrainingSet(200) if record else None
    if record:
        sim.record(data)
        extra.append(data)
    out = {}
    sim.begin3d()
    for s in sp:
        converge(s)
    sim.slices(c.nz)
    out["np"] = [s.np() for s in sp]
    st = sim.end3d()
    for name in ("bexyz", "bbxyz"):
        out[name] = sim.get_3d(name)
    out["q3"] = np.stack([sum(s.get_q3(l) for s in sp) for l in range(1, c.nz + 2)])
    out["epw"] = sim.get_field("epw")
    if record:
        out["pairs"] = [data.get(i) for i in range(len(data))]
    for h in [sim, bm, *sp, *extra, c]:
        h.close()
    return st.regrowths, out


@pytest.mark.parametrize("kw", [dict(), dict(graphs=True), dict(nspecies=2),
                                dict(nspecies=2, graphs=True), dict(predict=3),
                                dict(predict=3, graphs=True), dict(record=True)],
                         ids=lambda kw: "-".join(kw) or "plain")
def test_step_that_overflows_is_the_step_with_room(qp, kw):
    grown, a = step(qp, 0.01, **kw)
    none, b = step(qp, 6.0, **kw)
    assert grown > 0 and none == 0
    assert a["np"] == b["np"]
    for name in ("bexyz", "bbxyz", "q3", "epw"):
        assert rel_l2(a[name], b[name]) < 1e-4, (name, rel_l2(a[name], b[name]))
    if "pairs" in b:  # one pair per slice, none of them recorded twice
        assert len(a["pairs"]) == len(b["pairs"]) == 32
        for (xa, ta, sa), (xb, tb, sb) in zip(a["pairs"], b["pairs"]):
            # features are rounded to bfloat16 (2^-8), targets are differences of
            # the passes' iterates over their scale
            assert np.isclose(sa, sb, rtol=1e-3)
            assert rel_l2(xa, xb) < 1e-2 and np.abs(ta - tb).max() < 1e-2 + 1e-2 * np.abs(tb).max()


@pytest.mark.parametrize("graphs", [False, True])
def test_a_failed_network_ends_the_step(qp, graphs):
    """The error flag that a network's kernel raises when a wait expires (set
    here from the host) reaches the caller of the step, and a cleared one does
    not."""
    c = qp.Context(7, 7, 3, BOX)
    sp = qp.Species2d(c, ppc=(2, 2))
    bm = qp.Beam3d(c, (16, 16, 16), peak_density=1.0, center=(0.0, 0.0, 2.5),
                   sigma=(0.5, 0.5, 0.5))
    sim = qp.Simulation(c, [sp], [bm], iter=2, predict=3, use_graphs=graphs)
    net = qp.Predictor(seed=1)
    sim.set_predictor(net)
    sim.step3d()
    want = sim.get_3d("bexyz")
    assert qp.lib().qp_nn_flag_error(net.h, 1) == 0
    with pytest.raises(qp.QPError, match="learned start: a bounded wait"):
        sim.step3d()
    with pytest.raises(qp.QPError, match="bounded wait expired"):
        net.forward(np.zeros((1, 16, 1, 128), dtype=np.float32))
    assert qp.lib().qp_nn_flag_error(net.h, 0) == 0
    sp.renew(0.0)  # the failed step has moved the particles
    sim.step3d()
    assert rel_l2(sim.get_3d("bexyz"), want) < 1e-5
    for h in (sim, net, bm, sp, c):
        h.close()
