"""What several host threads may share."""
import threading

import numpy as np
import pytest
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qp():
    import qpgpu

    return qpgpu


def run_threads(work):
    """Every callable of `work` in a thread of its own, started together; an
    exception in any of them fails the test."""
    start, errors = threading.Barrier(len(work)), []

    def body(f):
        try:
            start.wait(60)
            f()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=body, args=(f,)) for f in work]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]


# one shape for all threads (shared work buffers), and one each (every call
# finds the buffers of another shape)
@pytest.mark.parametrize("shapes", [[(2, 9, 128)] * 3, [(1, 5, 128), (2, 7, 256), (3, 3, 128)]])
def test_threads_take_turns_on_one_network(qp, shapes):
    """The network's work buffers belong to one call at a time: what a thread
    gets is what it gets alone.  The forward pass has no sum whose order
    changes, so it is exact; the gradient is summed by reductions in any order
    (FP32, 1e3 to 1e4 terms: 1e-5)."""
    rng = np.random.default_rng(4)
    net = qp.Predictor(seed=3)
    net.set_params(rng.normal(0, 0.1, net.nparams).astype(np.float32))
    jobs = []
    for nb, h, w in shapes:
        x = rng.normal(0, 1, (nb, 16, h, w)).astype(np.float32)
        t = rng.normal(0, 1, (nb, 2, h, w)).astype(np.float32)
        jobs.append((x, t, net.forward(x), *net.loss_grad(x, t)))

    def work(x, t, out, loss, grad):
        for _ in range(10):
            assert np.array_equal(net.forward(x), out)
            l, g = net.loss_grad(x, t)
            assert abs(l - loss) < 1e-5 * loss and rel_l2(g, grad) < 1e-5

    run_threads([lambda j=j: work(*j) for j in jobs])
    net.close()


def host_buffers(qp):
    import ctypes as C

    bytes_, pinned = C.c_longlong(), C.c_longlong()
    assert qp.lib().qp_host_buffers(C.byref(bytes_), C.byref(pinned)) == 0
    return bytes_.value, pinned.value


def test_one_context_after_another_pins_once(qp):
    def cycle():
        c = qp.Context(5, 5, 2, [[-6.0, 6.0], [-6.0, 6.0], [0.0, 1.0]])
        f = qp.Field2d(c, 3)
        f.as_(2.0)
        assert (f.get_rs()[:, :, : c.ny + 1] == 2.0).all()
        f.close()
        c.close()

    cycle()
    bytes0, pinned0 = host_buffers(qp)
    for _ in range(5):
        cycle()
    assert host_buffers(qp) == (bytes0, pinned0) and bytes0 > 0


def test_threads_with_a_context_each_transfer_at_once(qp):
    """Each transfer has its own pair of host buffers; afterwards no more of
    them are kept than the bound says.  Values are only moved: exact."""
    def work(k):
        c = qp.Context(7, 7, 3, [[-6.0, 6.0], [-6.0, 6.0], [0.0, 1.0]])
        f = qp.Field2d(c, 3)
        rng = np.random.default_rng(k)
        for _ in range(8):
            a = rng.standard_normal(c.ks_shape(3)).astype(np.float32)
            f.set_ks(a)
            assert np.array_equal(f.get_ks(), a)
        f.close()
        c.close()

    run_threads([lambda k=k: work(k) for k in range(8)])
    assert host_buffers(qp)[0] <= 4 * 512 * 1024
