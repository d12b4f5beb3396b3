"""The even-odd phase timers accumulate over solves, with either kernel: a second
solve of the same sources (the same iterations, bit for bit) doubles every count."""
import ctypes as C

import numpy as np
import pytest

from conftest import quenched_theta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [-1, 0])
def test_phase_counts_add_up(kernel):
    import three_part_dwf_study_b200 as T
    from three_part_dwf_study_b200 import _capi as A
    rng = np.random.default_rng(7)
    d = T.DomainWall(16, 12, 8, 1.0, 0.1)
    d.set_gauge(quenched_theta(rng, 16, 12, 3.0))
    A.check(A.lib().dwf_set_eo_kernel(d.handle, kernel), d.handle)
    src = rng.normal(size=(3, d.Ndof)) + 1j * rng.normal(size=(3, d.Ndof))
    A.check(A.lib().dwf_eo_phase_profile(d.handle, 1), d.handle)
    ms, cnt, seen = (C.c_double * 8)(), (C.c_uint64 * 8)(), []
    for _ in range(2):
        d.propagators(src, rtol=1e-10, maxiter=20000, solver=T.SOLVER_EO_MIXED)
        A.check(A.lib().dwf_eo_phase_times(d.handle, ms, cnt), d.handle)
        seen.append((np.array(cnt), np.array(ms)))
    assert seen[0][0][0] > 0 and np.array_equal(seen[1][0], 2 * seen[0][0])
    assert (seen[1][1][:7] > seen[0][1][:7]).all()
    d.close()
