"""sl_trait_backward with no graphs and no gradient of log P(T) asked for leaves
what is queued, and the status that it reports, to the next call that waits."""
import ctypes

import numpy as np
import pytest

from conftest import load_golden
from swiftlink_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


def test_status_stays():
    torch = pytest.importorskip("torch")
    g = load_golden("cfg1")
    g["disease_prob"] = np.array(g["disease_prob"])
    g["disease_prob"][g["N"] - 1] = 0.0   # nobody can be as the last member is: every position's likelihood is 0
    words = g["M"] * ((2 * (g["N"] - g["F"]) + 31) // 32)
    with api.Context(api.Problem.from_arrays(g), n_chains=1) as ctx:
        graph = torch.zeros(words, dtype=torch.int32, device="cuda")
        acc = torch.zeros((g["M"] - 1) * g["n_lod"], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        fn = api.lib().sl_lod_score_device_graphs_noalloc
        fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
        assert fn(ctx.h, 1, graph.data_ptr(), acc.data_ptr()) == api.SL_OK
        torch.cuda.synchronize()
        assert api.lib().sl_trait_backward(ctx.h, 0, None, None, None) == api.SL_OK
        with pytest.raises(api.SwiftLinkError) as e:
            ctx.synchronize()
        assert e.value.code == api.SL_EZERO
