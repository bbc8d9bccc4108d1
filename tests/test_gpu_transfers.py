"""Arrays in the caller's layouts, to and from the device planes: the conversion
runs on the device, in parts of 2^16 values through two pinned halves, so the
sizes below fall short of, on and past the edges of a part and of a pair of
parts.  Values are only moved: every comparison is exact."""
import numpy as np
import pytest
from conftest import BOX

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qp():
    import qpgpu

    return qpgpu


@pytest.mark.parametrize("np_", [1, 9362, 9363, 18724, 18725, 1300001])
def test_beam_particles_round_trip(qp, np_):
    c = qp.Context(5, 5, 3, BOX)
    b = qp.Beam3d(c, (np_, 1, 1), quiet_start=False, sigma=(0.5, 0.5, 0.5), center=(0, 0, 5.0))
    rng = np.random.default_rng(np_)
    p = np.asfortranarray(rng.uniform(2, 6, (7, np_)).astype(np.float32))
    b.set_particles(p)
    assert np.array_equal(b.get_particles(), p)
    b.close()
    c.close()


@pytest.mark.parametrize("ind", [(4, 4), (6, 9), (10, 10)])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_fields_round_trip(qp, ind, dim):
    c = qp.Context(ind[0], ind[1], 1, BOX)
    f = qp.Field2d(c, dim)
    rng = np.random.default_rng(dim)
    rs = rng.standard_normal(c.rs_shape(dim)).astype(np.float32)
    ks = rng.standard_normal(c.ks_shape(dim)).astype(np.float32)
    f.set_rs(rs)
    f.set_ks(ks)
    got = f.get_rs()
    assert np.array_equal(got[:, :, : c.ny + 1], rs[:, :, : c.ny + 1])
    assert not got[:, :, c.ny + 1:].any()  # rows past the guard row
    assert np.array_equal(f.get_ks(), ks)
    f.close()
    c.close()


@pytest.mark.parametrize("ind", [(5, 4, 4), (7, 7, 7)])
def test_whole_arrays_are_their_planes(qp, ind):
    c = qp.Context(*ind, BOX)
    sp = qp.Species2d(c, ppc=(2, 2))
    bm = qp.Beam3d(c, (16, 16, 16), peak_density=2.0, center=(0, 0, 3.0), sigma=(0.5, 0.5, 0.5))
    sim = qp.Simulation(c, [sp], [bm], iter=1, vpot=True)
    sim.begin3d()
    sim.slices(c.nz - 1)
    pp, kp = sp.get_particles()
    assert kp.sum() == sp.np()
    for t in (0, len(kp) // 2, len(kp) - 1):
        assert not pp[:, kp[t]:, t].any() and (pp[7, : kp[t], t] != 0).all()
    ld = pp.shape[1] + 3  # another leading dimension, another tile pitch
    wide, _ = sp.get_particles(ld)
    assert np.array_equal(wide[:, : pp.shape[1]], pp) and not wide[:, pp.shape[1]:].any()
    sp.set_particles(wide, kp)
    assert np.array_equal(sp.get_particles()[0], pp)
    sim.slices(1)
    for name in ("bexyz", "bbxyz", "vpot", "q3"):
        whole = sim.get_3d(name)
        for l in (0, 1, c.nz // 2, c.nz):
            assert np.array_equal(whole[..., l], sim.get_plane(name, l)), name
    q = bm.get_q3d()
    for l in (0, c.nz // 3, c.nz):
        assert np.array_equal(q[..., l], sim.get_plane("qb", l))
    sim.end3d()
    for h in (sim, bm, sp, c):
        h.close()


def test_transfers_run_on_their_contexts_device(qp):
    """Reading and writing a context's arrays while another device is current."""
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    c = qp.Context(5, 5, 1, BOX, device=0)
    sp, f = qp.Species2d(c, ppc=(2, 2)), qp.Field2d(c, 2)
    other = qp.Context(5, 5, 1, BOX, device=1)  # makes device 1 the current one
    a = np.random.default_rng(1).standard_normal(c.ks_shape(2)).astype(np.float32)
    f.set_ks(a)
    assert np.array_equal(f.get_ks(), a)
    pp, kp = sp.get_particles()
    sp.set_particles(pp, kp)
    assert np.array_equal(sp.get_particles()[0], pp)
    for h in (f, sp, c, other):
        h.close()
