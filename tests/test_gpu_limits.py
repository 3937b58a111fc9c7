"""Limits that a call states or meets: the caller's round cap."""
import numpy as np
import pytest

import dynamicssspv2_gb300 as D
from tests.common import check_against_oracle

pytestmark = pytest.mark.gpu


def _i32(*arrays):
    return tuple(np.ascontiguousarray(x, np.int32) for x in arrays)


def _spine_and_chain(spine, leaves, chain):
    """A tree from vertex 0: a spine each of whose vertices carries that many leaves, beside a bare
    chain; its edges (the first of the spine and of the chain are lines 0 and 1) and its depth."""
    s = 1 + np.arange(spine)
    c = 1 + spine + np.arange(chain)
    at = 1 + spine + chain
    u = np.concatenate([[0, 0], s[:-1], c[:-1], np.repeat(s, leaves)])
    v = np.concatenate([[s[0], c[0]], s[1:], c[1:], at + np.arange(spine * leaves)])
    n = at + spine * leaves
    w = 1 + (np.arange(len(u)) * 2654435761 % 5)
    return n, *_i32(u, v, w), max(spine + 1, chain)


@pytest.mark.parametrize("opts", [{}, {"warp_agg": 1}, {"small_deg": 16}, {"solo_waves": 0}, {"group_ctas": 4}], ids=str)
@pytest.mark.parametrize("spine,leaves,chain", [(90, 40, 200), (200, 40, 90), (120, 3, 120), (1, 40, 300)])
def test_a_round_cap_counts_rounds(spine, leaves, chain, opts):
    """In a tree every vertex is reached once, in the round of its depth: a cap of depth + 1 rounds is
    enough for the computation from the root whatever runs beside it (a spine of long rows goes one
    vertex a list, the chain hundreds of steps in a queue), one less is not; the same for a batch
    that joins both branches to the root, which begins one level below."""
    n, u, v, w, depth = _spine_and_chain(spine, leaves, chain)
    n += 64 * spine  # isolated vertices: rows are short on the whole
    join = D.make_changes(u[:2], v[:2], w[:2], np.ones(2))

    def capped(cap, first):
        return D.Graph(n, u[first:], v[first:], w[first:], max_rounds=cap, recover=0, **opts)

    with capped(depth + 1, 0) as g:
        for _ in range(3):
            assert g.tree_compute(0).rounds == depth + 1
        p, d = g.tree_read()
        check_against_oracle(n, u, v, w, None, 0, p, d, "tree under a cap")
    with capped(depth, 0) as g:
        with pytest.raises(D.DsssspError) as e:
            g.tree_compute(0)
        assert e.value.code == D.E_NO_CONVERGENCE
    with capped(depth, 2) as g:
        g.tree_compute(0)
        g.snapshot()
        for _ in range(3):
            g.restore()
            assert g.apply_batch(join).rounds == depth
        p, d = g.tree_read()
        check_against_oracle(n, u, v, w, None, 0, p, d, "batch under a cap")
    with capped(depth - 1, 2) as g:
        g.tree_compute(0)
        with pytest.raises(D.DsssspError) as e:
            g.apply_batch(join)
        assert e.value.code == D.E_NO_CONVERGENCE


def test_a_round_cap_on_near_far_rounds():
    """Under a cap near-far rounds are counted one by one too: what a capped call needed is enough for
    the next, one less is not, and a cap that no computation passes changes nothing."""
    n, u, v, w, depth = _spine_and_chain(60, 40, 400)
    with D.Graph(n, u, v, w, delta=20, recover=0, max_rounds=2 * n) as g:
        need = g.tree_compute(0).rounds
        assert depth < need <= 2 * depth
        o = g.get_opts()
        for cap, good in ((need, True), (need - 1, False), (need, True), (2 * n + 16, True)):
            o.max_rounds = cap
            g.set_opts(o)
            if good:
                st = g.tree_compute(0)
                assert st.rounds <= need or cap == 2 * n + 16
                p, d = g.tree_read()
                check_against_oracle(n, u, v, w, None, 0, p, d, f"cap {cap}")
            else:
                with pytest.raises(D.DsssspError) as e:
                    g.tree_compute(0)
                assert e.value.code == D.E_NO_CONVERGENCE
