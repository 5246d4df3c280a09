"""Several host threads assembling on builders of their own, of different orders: their launches ask
for different amounts of shared memory of the same kernels.  Every call succeeds and gives what it
gives alone, for one mesh a launch and for several."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from helmholtzbem_gb300 import api, geometry  # noqa: E402


def run(work, rounds):
    alone = [f() for f in work]
    bad = []

    def go(f, ref):
        try:
            for _ in range(rounds):
                if not np.array_equal(f(), ref):
                    bad.append("another result")
                    return
        except Exception as e:   # noqa: BLE001
            bad.append(str(e))
    ts = [threading.Thread(target=go, args=w) for w in zip(work, alone)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[0]


def test_layers_of_builders_of_different_orders():
    def work(order):
        b = api.GalerkinBuilder(api.BuilderData(geometry.circle(0.25, 12), order=order))

        def f():
            for _ in range(10):   # little but launches: the threads meet between asking and launching
                b.assembleDense(2.0, 3.0, d=2)
            return np.stack([b.getDoubleLayer(2), b.getHypersingular(1), b.getSingleLayer(0)])
        return f
    run([work(o) for o in (16, 11, 20, 7)], 200)


def test_several_meshes_in_one_launch():
    def work(orders):
        ops = [api.SolutionsOperator(api.BuilderData(geometry.circle(0.2, 6 + o), order=o)) for o in orders]

        def f():
            for _ in range(10):
                T = api.gen_sol_op_multi_device(ops, [[1.0, 2.5]] * len(ops), 1.0, [4.0] * len(ops), d=2)
            return np.concatenate([np.asarray(t.cpu()).ravel() for t in T])
        return f
    run([work(o) for o in ((2, 3), (20, 11), (7, 16))], 100)
