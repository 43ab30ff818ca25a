"""A population index outside [0, P) anywhere among a call's indices is refused."""
from __future__ import annotations

import numpy as np
import pytest

from steppecu_b200 import F2Tensor, StpError, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0, 1, 17, 398, 399])
@pytest.mark.parametrize("bad", [-1, 5, 2**31 - 1, -(2**31)])
def test_index_outside_is_refused(ctx, at, bad):
    P, nb = 5, 3
    t = F2Tensor(np.full(P * P * nb, 0.25), np.full(P * P * nb, 9.0), np.full(nb, 40, np.int32), P, nb)
    q = np.arange(400, dtype=np.int32) % P
    assert ctx.f4(t, q.reshape(-1, 4))[2] == nb
    q[at] = bad
    with pytest.raises(StpError, match="outside") as e:
        ctx.f4(t, q.reshape(-1, 4))
    assert e.value.status == _lib.STP_INVALID_ARGUMENT
