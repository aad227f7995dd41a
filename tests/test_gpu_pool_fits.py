"""Single calls run into what the device's shared workspace holds. A call like the one before
it fits, whatever its lists' entries take: it enqueues what a batch's run enqueues, once."""
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu

OPTIONS = {"exact": dict(), "mixed": dict(precision=1), "plain": dict(precision=2), "brick8": dict(brick=8),
           "brick4": dict(brick=4), "mixed4": dict(brick=4, precision=1)}


@pytest.mark.parametrize("size", [(2, 30), (4, 90)])
def test_a_repeated_call_runs_once(cm, size):
    plc = cm.PLC.from_arrays(*W.jittered_icosphere(size[0], 0.03, seed=1))

    def launches(f):
        n = cm.gpu_launches()
        f()
        return cm.gpu_launches() - n

    once = {}
    for name, kw in OPTIONS.items():
        b = cm.Batch([plc], [size[1]], [1], outputs=3, **kw)
        b.run().sync()
        once[name] = launches(lambda: b.run().sync())
    for name, kw in (*OPTIONS.items(), *reversed(OPTIONS.items())):
        def call():
            return cm.voxelize_ex(plc, resolution=size[1], pad=1, outputs=3, **kw)
        call()
        assert launches(call) == once[name] and launches(call) == once[name], name
