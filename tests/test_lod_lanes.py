"""The FP64 trait peel with several positions to a warp: few and many positions
(two lane counts), a last warp that is not full, cutsets of up to three
members, the plain and the rescaled form."""
import numpy as np
import pytest

from conftest import load_golden
from swiftlink_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


# positions per graph: loop 10, east 495; 20,000 and more take the narrower form
@pytest.mark.parametrize("name,graphs", [("loop", 1), ("loop", 2001), ("east", 1), ("east", 39), ("east", 42)])
@pytest.mark.parametrize("precision", [api.SL_LOD_FP64, api.SL_LOD_FP64_RESCALED])
def test_table_of_repeated_graphs(name, graphs, precision):
    g = load_golden(name)
    n = g["lod_graphs"].shape[0]
    stack = g["lod_graphs"][np.arange(graphs) % n]
    with api.Context(api.Problem.from_arrays(g), n_chains=1, lod_precision=precision) as ctx:
        ctx.lod_score_graphs(stack)
        raw, cnt, tp = ctx.lod_results()
    assert cnt == graphs
    if graphs % n:   # the golden table is of whole sets; a part of one by the oracle
        from oracle import port
        want = api.lod_table(*port.Port(g).lod(stack))
    else:
        want = api.lod_table(g["lod_raw"], g["lod_count"], g["lod_trait_prob"])
    assert np.abs(api.lod_table(raw, cnt, tp) - want).max() <= 1e-10
