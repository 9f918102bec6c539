"""The near pairs' kernel shares its work between the SMs that it gets: the
far and on-element kernels beside it may hold any of them when it starts."""
import numpy as np
import pytest

from bem_gmsh_gb300 import _lib, star_domain
from bem_gmsh_gb300.api import solve

pytestmark = pytest.mark.gpu


def test_every_pair_near_takes_the_same_time_each_call():
    dad = star_domain(333, p=2, seed=3)
    ctx = _lib.Context()
    try:
        t = []
        for _ in range(40):
            _, st = solve(dad, npg=8, near_factor=np.inf, ctx=ctx, return_stats=True)
            t.append(st["t_assemble_ms"])
        t = np.sort(t[3:])
        # half of the SMs without a task would double it
        assert t[-3] <= 1.4 * t[0], t
    finally:
        ctx.close()
