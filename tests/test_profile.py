"""moist_step_profile: the kernels it counts in each group of the large step."""
import ctypes as C

import numpy as np
import pytest

from moist2d_b200 import abi, model
from moist2d_b200._lib import lib
from states import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags,sweep", [(0, 1), (abi.MOIST_FLAG_TRACER_DATAFLOW, 2), (abi.MOIST_FLAG_TRACER_STREAM, 2),
                                         (abi.MOIST_FLAG_TRACER_WAVEFRONT, 1)],
                         ids=["tiles", "dataflow", "stream", "wavefront"])
def test_launches_by_group(flags, sweep):
    """Kernels a step: the tiled sweep is one launch a stage, its dataflow form is followed by the count of
    its computations, the streaming sweep is preceded by its records."""
    p, s = small_case(np.float32, 48, 20, do_sf=True, do_rd=True)
    steps = 2
    n = (C.c_longlong * abi.MOIST_NGROUPS)()
    with model.Model(p, flags) as m:
        m.upload(s)
        rc = lib().moist_step_profile(m.ctx, steps, C.byref(C.c_float()), (C.c_float * abi.MOIST_NGROUPS)(), n)
    assert rc == abi.MOIST_OK
    subs = -(-p.ns // 3) + -(-p.ns // 2) + p.ns
    # physics, prologue, substep, tracer, update, other
    assert list(n) == [steps * k for k in (3, 9, subs, 3 * sweep, 6, 1)]
