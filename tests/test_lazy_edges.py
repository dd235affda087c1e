"""Lazy check at the sizes its kernels switch or split at: candidates per node
around what a warp sorts (512) and around a power of two, nodes around the tiles
of 256, fewer candidates than the lanes of a node.  Every primitive is in the
ball; the accepted set and the checks are those of the oracle (exact)."""
import dataclasses

import numpy as np
import pytest

import oracle_bind as ob
from dynoplan_gb300 import workloads as W
from lazy_ref import lazy_accept
from test_lazy import run_lazy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,P,limit", [(1, 8, 3), (255, 9, 20), (257, 64, 1), (33, 129, 20), (300, 511, 7),
                                       (20, 512, 20), (20, 513, 20), (2049, 70, 9)])
@pytest.mark.parametrize("score_kind", ["random", None])
def test_lazy_sizes(N, P, limit, score_kind):
    wl = dataclasses.replace(W.make_workload(2, seed=31 + P, N=N, P=P), delta=1e3)
    ball, score, got, st, _lib = run_lazy(wl, 0, limit, score_kind, seed=N)
    assert ball["n_pairs"] == N * P and st["max_candidates"] == P
    ora = ob.expand(wl.robot, wl.prims, wl.env, wl.nodes, wl.radius, fast=True, threads=ob.lib().orc_max_threads())
    key = lambda r: r["node"].astype(np.int64) * P + r["prim"].astype(np.int64)
    valid = np.zeros(N * P, bool)
    valid[key(ora)] = ora["verdict"] == 0
    valid = valid[key(ball)]
    accepted, needed = lazy_accept(ball["node"], ball["prim"], valid, score, limit)
    checked = got["verdict"] != _lib.DPG_UNCHECKED
    np.testing.assert_array_equal((got["flags"] & _lib.DPG_FLAG_ACCEPTED) != 0, accepted)
    np.testing.assert_array_equal(got["verdict"][checked] == 0, valid[checked])
    assert checked[needed].all()
    assert st["n_checked"] == int(checked.sum()) and st["n_accepted"] == int(accepted.sum())
    assert st["n_valid"] == int((got["verdict"] == 0).sum())


def test_lazy_many_nodes():
    """More than 8,192 nodes: the scan over the nodes' counts takes several passes."""
    test_lazy_sizes(20001, 20, 5, "random")
