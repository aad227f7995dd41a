"""A sizing field whose first evaluation meets a failed device allocation (made on the
host, cmg_debug_fail_device_allocs; no GPU fault is involved): the call answers "out of
memory", whichever of its buffers could not be had, and the field's next evaluation works
and gives the values of a field that never met one."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture()
def fail(cm):
    from cybermeshgenerator_gb300 import _lib
    L = _lib.load()

    def set_(skip, count):
        assert L.cmg_debug_fail_device_allocs(skip, count) == 0
    yield set_
    L.cmg_debug_fail_device_allocs(0, 0)


# the host call's three buffers, six per-query ones and the counting sort's four
@pytest.mark.parametrize("n,buffers", [(700, 13), (9000, 13)])
def test_first_evaluation_after_a_failed_allocation(cm, fail, n, buffers):
    P, T = W.kuhn_tet_mesh(5, 0.3, seed=5)
    S = np.random.default_rng(5).uniform(0.05, 1.0, len(P))
    Q = W.sizing_queries(P, T, n, seed=n)
    want, wwhich = cm.SizingField(P, T, S, 0.5).eval(Q, which=True)
    for skip in range(buffers):
        f = cm.SizingField(P, T, S, 0.5)
        fail(skip, 1)
        with pytest.raises(RuntimeError, match="out of memory"):
            f.eval(Q, which=True)
        fail(0, 0)
        for q, w, i in ((Q, want, wwhich), (Q[: n // 3], want[: n // 3], wwhich[: n // 3])):
            got, which = f.eval(q, which=True)
            assert np.array_equal(got.view(np.uint64), w.view(np.uint64)) and np.array_equal(which, i)
        f.close()
