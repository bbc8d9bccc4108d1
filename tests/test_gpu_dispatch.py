"""Where a size chooses between two forms of a kernel.

* Current deposit of the fused step: two CTAs per tile and 2 particles per
  thread up to 222 tiles, one and 4 beyond; tiles with less than one round of
  particles, exactly one, and more.  One 3D step on each side of the line,
  against the FP64 oracle; the bar is that of the whole-step tests (1e-4).
* Re-bin: up to 256 movers into a tile are placed by rank, up to 1024 sorted in
  shared memory, more in the inbox.  Values are only moved, so the tiles must
  hold exactly the particles they should, the movers in cell order.
* A step at 8 x 8 particles per cell, whose inboxes (19661 slots of a tile) are
  larger than any sort in shared memory.
"""
import numpy as np
import pytest
from conftest import make_config, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qp():
    import qpgpu

    return qpgpu


def step_against_oracle(qp, oracle_mod, ind, ppc):
    cfg = make_config(ind=ind, ppc=ppc, iter=2)
    b = cfg["beams"][0]
    c = qp.Context(*ind, cfg["grid"]["box"])
    sp = qp.Species2d(c, ppc=ppc)
    bm = qp.Beam3d(c, b["np"], q=b["q"], m=b["m"], gamma=b["gamma"], quiet_start=True,
                   peak_density=b["peak_density"], center=b["center"], sigma=b["sigma"])
    sim = qp.Simulation(c, [sp], [bm], iter=2)
    sim.step3d()
    o = oracle_mod.Sim(cfg, np.float64)
    o.begin3d()
    for j in range(1, (1 << ind[2]) + 1):
        o.slice(j)
    for name in ("bexyz", "q3"):
        got = sim.get_3d(name)
        assert rel_l2(got, o.get(name).reshape(got.shape, order="F")) < 1e-4, name
    for h in (sim, bm, sp, c):
        h.close()


# every length of line in x and in y, where the transforms, their register
# caps and the staging of the x passes and column solves differ
@pytest.mark.parametrize("ind", [(10, 5, 4), (5, 10, 4), (11, 4, 4), (4, 11, 4), (7, 8, 4), (8, 7, 4)])
def test_step_at_every_line_length(qp, oracle_mod, ind):
    step_against_oracle(qp, oracle_mod, ind, (2, 1))


# 1 tile; 64; 128 tiles (two CTAs each); 256 (one); ppc 1, 4 and 6 per cell:
# 256, 1024 and 1536 particles per tile
@pytest.mark.parametrize("ind,ppc", [((4, 4, 4), (2, 2)), ((5, 9, 4), (1, 1)), ((8, 7, 4), (3, 2)),
                                     ((8, 8, 4), (1, 1)), ((8, 8, 4), (3, 2)), ((5, 5, 4), (8, 8))])
def test_step_on_both_sides_of_the_tile_count_rule(qp, oracle_mod, ind, ppc):
    step_against_oracle(qp, oracle_mod, ind, ppc)


# 16, 256, 320, 560, 1024, 1040, 4608 movers
@pytest.mark.parametrize("ppc", [(1, 1), (4, 4), (4, 5), (5, 7), (8, 8), (5, 13), (16, 18)])
def test_rebin_places_any_number_of_movers(qp, ppc):
    c = qp.Context(6, 6, 1, [[-6.0, 6.0], [-6.0, 6.0], [0.0, 1.0]])
    sp = qp.Species2d(c, ppc=ppc)
    pp, kp = sp.get_particles()
    for t in range(len(kp)):
        pp[0, : kp[t], t] += 1.0  # one column of cells per tile moves on
        pp[4, : kp[t], t] = np.arange(kp[t])  # a mark of its own
    pp[2] = np.arange(len(kp), dtype=np.float32)[None, :]  # and the tile it came from
    before = np.concatenate([pp[:, : kp[t], t] for t in range(len(kp))], axis=1)
    before[0] %= c.nx
    sp.set_particles(pp, kp)
    sp.pmove()
    qq, kq = sp.get_particles()
    after = np.concatenate([qq[:, : kq[t], t] for t in range(len(kq))], axis=1)
    order = lambda a: a[:, np.lexsort((a[4], a[2]))]  # noqa: E731
    assert np.array_equal(order(after), order(before))
    most = 0
    for t in range(len(kq)):
        x, y = qq[0, : kq[t], t].astype(int), qq[1, : kq[t], t].astype(int)
        assert ((x // 16) + 4 * (y // 16) == t).all()
        new = qq[2, : kq[t], t] != t
        most = max(most, int(new.sum()))
        if new.any():
            first = int(np.argmax(new))
            assert new[first:].all()  # the movers follow the stayers
            cell = (y[first:] % 16) * 16 + x[first:] % 16
            assert (np.diff(cell) >= 0).all()
    assert most == 16 * ppc[0] * ppc[1]
    sp.close()
    c.close()
