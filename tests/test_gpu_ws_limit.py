"""A one-launch Hessenberg basis whose exchange buffers (1.2 MB here) do not fit the workspace is built by the schedules
that need less, bit for bit the same.  The limit leaves room for the results and the other schedules' buffers (below
200 KB)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def limited(built_lib):
    from mixedprecisionofrr_gb300 import api

    ctx = api.context()

    def run(limit, call):
        ctx.lib.ofrr_debug_ws_limit(ctx.h, limit)
        try:
            ctx.reset_launch_count()
            out = call()
            return out, ctx.launch_count
        finally:
            ctx.lib.ofrr_debug_ws_limit(ctx.h, -1)

    return run


@pytest.mark.parametrize("m", [8192, 30000])
def test_falls_back_to_a_smaller_schedule(limited, m):
    from mixedprecisionofrr_gb300 import api

    rng = np.random.default_rng(m)
    n = 64
    A = rng.standard_normal((m, n)) @ rng.standard_normal((n, n))
    (Q0, R0, s0, p0), one = limited(-1, lambda: api.hessenberg(A, "double", "double"))
    (Q1, R1, s1, p1), many = limited(400_000, lambda: api.hessenberg(A, "double", "double"))
    assert many > one  # blocks or columns, a launch and more each
    assert np.array_equal(api.to_numpy(Q0), api.to_numpy(Q1)) and np.array_equal(R0, R1)
    assert np.array_equal(s0, s1) and np.array_equal(p0, p1)
    with pytest.raises(Exception):  # no room at all: the error, as before
        limited(1000, lambda: api.hessenberg(A, "double", "double"))
    (Q2, R2, _, _), again = limited(-1, lambda: api.hessenberg(A, "double", "double"))
    assert again == one and np.array_equal(R0, R2)
