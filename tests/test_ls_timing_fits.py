"""The L-sampler's timed choice on rfunctions so wide that two or four tasks'
arenas do not fit a block: those lane groups are left out."""
import numpy as np
import pytest

from swiftlink_gb300 import api
from test_refused_call import wide

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


def test_choice():
    g = wide()
    prob = api.Problem.from_arrays(g, with_legal=False)
    u = np.random.default_rng(1).random((1, g["M"], g["K"] + 2 * g["N"]))
    got = []
    for form in (api.SL_LS_KERNEL_GENERIC32, api.SL_LS_KERNEL_GENERIC):
        with api.Context(prob, ls_kernel=form) as ctx:
            ctx.set_graphs(g["dg0"])
            ctx.lsampler_sweep(u)
            got.append(ctx.get_graphs())
            lanes, times = ctx.ls_tuning()
    assert times[0] > 0 and times[2] == 0 and lanes in (32, 16, 4)   # four tasks take 320 KB
    assert np.array_equal(got[0], got[1])
