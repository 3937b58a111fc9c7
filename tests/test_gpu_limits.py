"""Limits that a call states or meets: the caller's round cap, the range of the distances,
the count of the entries, host memory that is pinned in part, device memory."""
import gc
import mmap

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


W = 1_500_000_000  # two of these fit a distance, three do not


def _late_long_paths(gates, light, leaves):
    """From vertex 1, behind vertex 0, `gates` pairs of paths to a vertex of their own each: a light one
    whose vertices carry leaves, and a bare one a hop longer that ends in three edges of W."""
    u, v, w, n = [[0]], [[1]], [[3]], 2
    take = lambda k: np.arange(n, n + k)  # noqa: E731
    ends = take(gates)
    n += gates
    prev = np.ones(gates, np.int64)
    for _ in range(light - 1):
        at = take(gates)
        n += gates
        u.append(prev), v.append(at), w.append(np.ones(gates))
        hang = take(gates * leaves)
        n += gates * leaves
        u.append(np.repeat(at, leaves)), v.append(hang), w.append(np.ones(len(hang)))
        prev = at
    u.append(prev), v.append(ends), w.append(np.ones(gates))
    prev = np.ones(gates, np.int64)
    for hop in range(light):
        at = take(gates)
        n += gates
        u.append(prev), v.append(at), w.append(np.full(gates, W if hop >= light - 2 else 1))
        prev = at
    u.append(prev), v.append(ends), w.append(np.full(gates, W))
    return n, *_i32(*(np.concatenate(x) for x in (u, v, w)))


@pytest.mark.parametrize("gates,opts", [(700, {"ctas_per_sm": 1}), (700, {}), (2000, {"warp_agg": 1}), (700, {"max_rounds": 400})],
                         ids=str)
def test_a_path_that_does_not_fit_beside_one_that_does(gates, opts):
    """Every distance fits, but an offer that does not may come first, by how far the CTAs' queues are: the
    computation and the batch that joins all of it to the root are not refused for it."""
    n, u, v, w = _late_long_paths(gates, 60, 12)
    join = D.make_changes(u[:1], v[:1], w[:1], np.ones(1))
    with D.Graph(n, u, v, w, **opts) as g:
        for _ in range(5):
            g.tree_compute(0)
        p, d = g.tree_read()
        check_against_oracle(n, u, v, w, None, 0, p, d, "tree")
    with D.Graph(n, u[1:], v[1:], w[1:], **opts) as g:
        g.tree_compute(0)
        g.snapshot()
        for _ in range(5):
            g.restore()
            g.apply_batch(join)
        p, d = g.tree_read()
        check_against_oracle(n, u[1:], v[1:], w[1:], join, 0, p, d, "batch")
        assert len(g.tree_read_changed()[0]) == n - 1


@pytest.mark.parametrize("opts", [{}, {"delta": 1000}, {"max_rounds": 8}], ids=str)
def test_a_distance_that_does_not_fit_is_refused(opts):
    """A vertex that only a path of more than 2^32 - 2 reaches: the computation, a batch that makes it so
    by a deletion or by an insertion and the call without allocation all report the overflow; what
    fits is exact, and the batch that mends it is accepted."""
    torch = pytest.importorskip("torch")
    u, v, w = _i32([0, 1, 2, 3, 0, 0], [1, 2, 3, 4, 4, 5], [W, W, W, 7, 9, 1])
    n = 6

    def refused(call, *args):
        with pytest.raises(D.DsssspError) as e:
            call(*args)
        assert e.value.code == D.E_OVERFLOW

    cut = D.make_changes(u[4:5], v[4:5], w[4:5], np.zeros(1))
    back = D.make_changes(u[4:5], v[4:5], w[4:5], np.ones(1))
    far = D.make_changes([2], [6], [1_400_000_000], [1])
    with D.Graph(n, u, v, w, **opts) as g:
        g.tree_compute(0)
        want = g.tree_read()
        assert list(want[1]) == [0, W, W + 16, 16, 9, 1]
        refused(g.apply_batch, cut)  # 3 and 4 only by three edges of W
        assert list(g.tree_read()[1]) == [0, W, 2 * W, -1, -1, 1]
        g.apply_batch(back)
        assert all(np.array_equal(a, b) for a, b in zip(g.tree_read(), want))
    with D.Graph(n + 1, u[[0, 1, 5]], v[[0, 1, 5]], w[[0, 1, 5]], **opts) as g:
        g.tree_compute(0)
        refused(g.apply_batch, far)
        assert list(g.tree_read()[1]) == [0, W, 2 * W, -1, -1, 1, -1]
    with D.Graph(n, u[[0, 1, 2, 5]], v[[0, 1, 2, 5]], w[[0, 1, 2, 5]], **opts) as g:
        refused(g.tree_compute, 0)
    off = torch.tensor([0, 1, 2, 3, 3], dtype=torch.int64, device="cuda")
    adj = torch.tensor([[1, W], [2, W], [3, W]], dtype=torch.int32, device="cuda")
    par = torch.empty(4, dtype=torch.int32, device="cuda")
    dist = torch.empty(4, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    refused(D.sssp_noalloc, 4, 3, off.data_ptr(), adj.data_ptr(), 0, par.data_ptr(), dist.data_ptr())
    adj[2, 1] = 2**31 - 1 - W  # 2 * W + that fits
    torch.cuda.synchronize()
    D.sssp_noalloc(4, 3, off.data_ptr(), adj.data_ptr(), 0, par.data_ptr(), dist.data_ptr())
    assert dist.tolist() == [0, W, 2 * W, W + 2**31 - 1]


def test_a_cut_off_vertex_beside_a_path_that_does_not_fit():
    """A pull sees every neighbour's offer: one that does not fit beside one that does is no overflow."""
    u, v, w = _i32([0, 1, 2, 0, 0], [1, 2, 3, 3, 3], [1_250_000_000, 1_250_000_000, 2 * 10**9, 10**9, 1_900_000_000])
    with D.Graph(4, u, v, w) as g:
        g.tree_compute(0)
        ch = D.make_changes(u[3:4], v[3:4], w[3:4], np.zeros(1))
        g.apply_batch(ch)
        p, d = g.tree_read()
        check_against_oracle(4, u, v, w, ch, 0, p, d, "pull")


def _regular(kind):
    if kind == "ring":
        a = np.arange(4096)
        return 4096, a, (a + 1) % 4096
    side = 96  # a torus: every row has four entries
    a = np.arange(side * side)
    y, x = a // side, a % side
    return side * side, np.concatenate([a, a]), np.concatenate([y * side + (x + 1) % side, (y + 1) % side * side + x])


@pytest.mark.parametrize("tails", [False, True])
@pytest.mark.parametrize("kind", ["ring", "torus"])
def test_lines_deleted_in_both_orientations_are_counted_once(kind, tails):
    """Rows of equal degree whose lines are deleted by many records of one batch, named from either end
    side by side: every entry is counted as one tombstone (tails: after the lines have come back by
    insertion, so that they lie in unsorted tails)."""
    n, u, v = _regular(kind)
    w = 1 + np.arange(len(u)) % 7
    u, v, w = _i32(u, v, w)
    gone = np.flatnonzero(np.arange(len(u)) % 8 != 0)
    a, b = u[gone], v[gone]
    both = D.make_changes(np.stack([a, b] * 4, 1).reshape(-1), np.stack([b, a] * 4, 1).reshape(-1), np.repeat(w[gone], 8),
                          np.zeros(8 * len(gone)))
    back = D.make_changes(a, b, w[gone], np.ones(len(gone)))
    with D.Graph(n, u, v, w, slack_pct=0, slack_min=8) as g:
        g.tree_compute(0)
        if tails:
            g.apply_batch(both)
            g.apply_batch(back)
        st = g.apply_batch(both)
        assert st.tombstoned == 2 * len(gone)
        assert g.health()["live"] == 2 * (len(u) - len(gone))
        p, d = g.tree_read()
        check_against_oracle(n, u, v, w, both, 0, p, d, kind)


PAGE = 1 << 16


@pytest.fixture
def patchwork():
    """Six pages of host memory, of which the first, the third and the fourth are pinned, each by itself."""
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    rt = torch.cuda.cudart()
    mem = np.frombuffer(mmap.mmap(-1, 7 * PAGE), np.uint8)
    mem = mem[-mem.ctypes.data % PAGE:][: 6 * PAGE]
    mem[:] = 77
    at = [mem.ctypes.data + k * PAGE for k in (0, 2, 3)]
    for p in at:
        assert int(rt.cudaHostRegister(p, PAGE, 0)) == 0
    yield mem
    torch.cuda.synchronize()
    for p in at:
        assert int(rt.cudaHostUnregister(p)) == 0


def test_a_failed_copy_is_reported_once(patchwork):
    """A read into an array that the runtime refuses to copy to fails alone: the next call is not told
    of it again."""
    torch = pytest.importorskip("torch")
    n = 3 * PAGE // 4
    u, v, w = D.gen_er(n, 2 * n, 1, 100, 5)
    with D.Graph(n, u, v, w) as g:
        g.tree_compute(0)
        want = g.tree_read32()
        with pytest.raises(D.DsssspError) as e:
            g.tree_read32_async(patchwork[: 4 * n].ctypes.data, None)  # a page of three is not pinned
        assert e.value.code == D.E_CUDA
        par, dist = (torch.empty(n, dtype=torch.int32).pin_memory().numpy() for _ in range(2))
        g.tree_read32(par, dist.view(np.uint32))
        assert np.array_equal(par, want[0]) and np.array_equal(dist.view(np.uint32), want[1])


def test_pinned_memory_is_pinned_throughout(patchwork):
    """Kernels read records from pinned memory and write trees to it only where all of the array is
    pinned, in one piece or in adjoining ones; an array with a pageable page between its pinned ends is
    left to the runtime's copy, which refuses it, and nothing is applied."""
    torch = pytest.importorskip("torch")
    n = PAGE // 4
    dist = torch.empty(n, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
    u, v, w = D.gen_er(n, 2 * n, 1, 100, 5)
    records = D.gen_changes(n, u, v, w, PAGE // 16, PAGE // 16, seed=6)  # two pages of them
    with D.Graph(n, u, v, w) as g:
        g.tree_compute(0)
        g.snapshot()
        want = g.tree_read32()
        whole = patchwork[2 * PAGE: 3 * PAGE].view(np.int32)
        g.tree_read32(whole, dist)
        assert np.array_equal(whole, want[0]) and np.array_equal(dist, want[1])
        across = patchwork[3 * PAGE - 2 * n: 3 * PAGE + 2 * n].view(np.int32)  # half in either pinned page
        g.tree_read32(across, dist)
        assert np.array_equal(across, want[0])
        patchwork[2 * PAGE: 4 * PAGE] = records.view(np.uint8)
        g.apply_batch(patchwork[2 * PAGE: 4 * PAGE].view(D.CHANGE_DTYPE))
        after = g.tree_read32()
        check_against_oracle(n, u, v, w, records, 0, *g.tree_read(), "records in two pinned pages")
        g.restore()
        gap = patchwork[PAGE // 2: 2 * PAGE + PAGE // 2]
        gap[:] = records.view(np.uint8)
        with pytest.raises(D.DsssspError) as e:
            g.apply_batch(gap.view(D.CHANGE_DTYPE))
        assert e.value.code == D.E_CUDA
        assert all(np.array_equal(a, b) for a, b in zip(g.tree_read32(), want))
        g.apply_batch(records)
        assert all(np.array_equal(a, b) for a, b in zip(g.tree_read32(), after))


def test_the_footprint_covers_what_a_graph_holds():
    """What a large sparse graph takes on the device once it has a tree and a batch behind it: the engine's
    own count of it and, without a spare region, which the estimate does not know of, the estimate by
    which tenants are admitted.  Allocations come in granules of 2 MiB; the lists of long rows'
    items (about 1.3 % of the slots at 48 bytes) are beside the estimate too."""
    torch = pytest.importorskip("torch")
    from dynamicssspv2_gb300.serve import estimate_footprint

    with D.Graph(100, *D.gen_er(100, 300, 1, 9, 1)) as g:  # modules are loaded, the context is up
        g.tree_compute(0)
        g.apply_batch(D.make_changes([1], [2], [3], [1]))
        g.tree_read()
    n, m = 1 << 23, 1 << 24
    u, v, w = D.gen_er(n, m, 1, 100, 7)
    ch = D.gen_changes(n, u, v, w, 500, 500, seed=8)
    gc.collect()  # graphs of other tests are gone
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with D.Graph(n, u, v, w, slack_pct=0, slack_min=4, spare_pct=0) as g:
        g.tree_compute(0)
        g.apply_batch(ch)
        used = before - torch.cuda.mem_get_info()[0]
        held = g.info()["device_bytes"]
        granules = 40 * (2 << 20)
        assert held <= used <= held + granules
        slots = 2 * m + 4 * n
        assert used <= estimate_footprint(n, m, 0, 4) + 0.013 * slots * 48 + granules
