"""All pairs in mixed precision at the sizes where the Hamaker kernel changes and at the edges of its 32-row tiles,
against the FP64 row kernel. Each row's FP32 terms (relative error about 3e-7) are added with compensation, so the
largest error of a field stays within 1e-6 of its largest value."""
import numpy as np
import pytest

from libgran_gb300 import _abi as A
from libgran_gb300 import configs as K
from libgran_gb300.system import System, generate_aggregate, generate_velocities

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hm", [A.LG_HAMAKER_LIMITED, A.LG_HAMAKER_FULL, A.LG_HAMAKER_SIMPLIFIED],
                         ids=["limited", "full", "simplified"])
@pytest.mark.parametrize("n", [2303, 2304, 2305, 2561])
def test_hamaker_over_all_pairs_equals_fp64(n, hm):
    mat = K.Material()
    x0, v0 = generate_aggregate(80, n, mat.r), generate_velocities(80, n, 0.1)
    acc = []
    for precision, kernel in ((A.LG_PRECISION_FP64, A.LG_FORCE_KERNEL_ROWGROUP), (A.LG_PRECISION_MIXED, A.LG_FORCE_KERNEL_AUTO)):
        d = K.make_desc(n, A.LG_BINARY_NONE, hm, hamaker=mat.hamaker(), precision=precision, force_kernel=kernel)
        s = System(d, x0, v0)
        acc.append(s.get(A.LG_FIELD_A))
        assert s.device_errors() == 0
        s.close()
    assert np.abs(acc[0]).max() > 0
    assert H.rel_err(acc[1], acc[0]) <= 1e-6
