"""The valid motions of a search's batch are collected from words of 64 motions
and 8 verdicts: motion counts around 64 and 128, pair counts of every remainder,
against the FP64 restatement (exact, as in test_search.py)."""
import pytest

from dynoplan_gb300 import workloads as W
from test_search import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 7, 63, 64, 65, 127, 129])
@pytest.mark.parametrize("batch", [1, 5])
def test_search_motion_words(dpg_lib, P, batch):
    import search_ref
    from dynoplan_gb300 import gpu as G
    from dynoplan_gb300 import search as S
    m, prims, env, start, goal = problem(W.UNICYCLE1, 40 + P, P=P, n_obs=6)
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        res, motions, _ = S.search(ctx, start, goal, S.options(0.9, batch=batch, max_expands=60, precision=1))
    ref = search_ref.search(m, prims, env, start, goal, 0.9, batch=batch, max_expands=60)
    assert (res["status_str"], res["expands"], res["nodes"]) == (ref["status"], ref["expands"], ref["nodes"])
    if ref["solved"]:
        assert list(motions) == ref["motions"]
