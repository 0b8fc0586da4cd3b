"""Sorted queries of large sets share walks of the tree
(k_knn_shared); queries in the given order are searched one by one.  Every
output of the two must have the same bits: the neighbour sets are exact and the
flux sums do not depend on the order of their terms."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from mnrt_b200 import _lib as L
from mnrt_b200 import gen
from mnrt_b200.batch import PhotonMapBatch
from mnrt_b200.photon_map import PhotonMap

pytestmark = pytest.mark.gpu


def to_dev(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def both(pm, qp, qn, nbr=True, **kw):
    """Outputs of the sorted and of the as-given query, which must agree bit for bit."""
    a = pm.query(qp, qn, want_nbr=nbr, **kw)
    b = pm.query(qp, qn, want_nbr=nbr, sorted_queries=False, **kw)
    torch.cuda.synchronize()
    for name in a:
        x, y = a[name].cpu().numpy(), b[name].cpu().numpy()
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), name
    return a


CASES = [
    # n, nq, k, R, filter, caustic, cluster, leaf (262,144 queries and more: walks are shared)
    (1, 262144, 1, 0.5, "box", 0.0, 0.0, 32),
    (2, 262145, 2, 2.0, "cone", 0.0, 0.0, 1),
    (40, 262151, 128, 3.0, "epanechnikov", 0.0, 0.0, 64),     # fewer photons than k
    (64, 262147, 1, 0.2, "cone", 0.0, 0.0, 64),
    (65, 262145, 31, 0.5, "cone", 0.0, 0.0, 64),
    (3000, 262150, 32, 0.1, "cone", 0.0, 0.0, 32),
    (3000, 262149, 33, 0.1, "epanechnikov", 0.2, 0.0, 7),
    (20000, 262145, 64, 0.05, "epanechnikov", 0.2, 0.5, 64),
    (100000, 262151, 65, 0.05, "cone", 0.2, 0.5, 32),
    (150000, 262145, 100, 0.1, "cone", 0.2, 0.0, 64),
    (50000, 262144, 128, 0.02, "box", 0.9, 0.5, 33),          # dense blob: queries left to the fix pass
    (30000, 262147, 8, 0.01, "cone", 0.2, 0.5, 64),           # R the bound of most queries
]


@pytest.mark.parametrize("nbr", [False, True])   # with lists, maps of few photons are searched one by one
@pytest.mark.parametrize("n,nq,k,r,filt,caustic,cluster,leaf", CASES)
def test_shared_walk_is_the_single_search(cuda, n, nq, k, r, filt, caustic, cluster, leaf, nbr):
    ph = gen.photons(n, seed=n + k, caustic_frac=caustic)
    q = gen.queries(nq, seed=nq, cluster_frac=cluster)
    q.pos[5 % nq, 0] = np.nan   # a query without a position in the middle of a group
    pm = PhotonMap(n, global_q_radius_max=r)
    pm.set_tuning(leaf_size=leaf)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    out = both(pm, to_dev(q.pos, cuda), to_dev(q.nrm, cuda), nbr, k=k, r_max=r, filter=filt, min_found=3)
    assert int(out["count"].max()) > 0
    assert pm.info().device_errors == L.PM_DEVERR_QNONFINITE


@pytest.mark.parametrize("copies", [2, 40, 1000])
def test_shared_walk_ties(cuda, copies):
    """Photons in `copies` places at once: the k-th distance is a tie of many."""
    n, nq, k = 4000, 262147, 50
    ph = gen.photons(n, seed=3, caustic_frac=0.0)
    ph.pos[:, :3] = np.tile(ph.pos[: n // copies, :3], (copies, 1))
    q = gen.queries(nq, seed=4)
    q.pos[:100, :3] = ph.pos[:100, :3]   # at distance 0 of a place
    pm = PhotonMap(n, global_q_radius_max=0.5)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    both(pm, to_dev(q.pos, cuda), to_dev(q.nrm, cuda), k=k, r_max=0.5, filter="cone")


@pytest.mark.parametrize("clump", [3, 5, 7, 11])
@pytest.mark.parametrize("nbr", [False, True])
def test_shared_walk_clumps(cuda, clump, nbr):
    """Queries in clumps apart by more than their radii: groups of 3, 5, 6 and 7
    that do not fit, halve, and grow back must still answer every query once."""
    n, k = 60000, 128
    ph = gen.photons(n, seed=8, caustic_frac=0.2)
    at = gen.queries(262144 // clump + 1, seed=9).pos[:, :3]
    rng = np.random.default_rng(clump)
    pos = np.zeros((len(at) * clump, 4), np.float32)
    pos[:, :3] = np.repeat(at, clump, 0) + rng.uniform(-0.02, 0.02, (len(at) * clump, 3)).astype(np.float32)
    nrm = np.zeros_like(pos)
    nrm[:, 1] = 1.0
    pm = PhotonMap(n, global_q_radius_max=0.2)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    both(pm, to_dev(pos, cuda), to_dev(nrm, cuda), nbr=nbr, k=k, r_max=0.2, filter="cone")


def test_shared_walk_in_a_batch(cuda):
    sizes = [(0, 50), (3, 700), (500, 1), (9000, 120001), (1, 60), (20000, 171345), (64, 0)]
    ks = [16, 128, 5, 64, 32, 100, 7]
    ph = [gen.photons(n, seed=10 + i, caustic_frac=0.2 if n > 100 else 0.0) for i, (n, _) in enumerate(sizes)]
    q = [gen.queries(m, seed=30 + i) for i, (_, m) in enumerate(sizes)]
    poff = np.concatenate([[0], np.cumsum([n for n, _ in sizes])])
    qoff = np.concatenate([[0], np.cumsum([m for _, m in sizes])])
    descs = [dict(k=k, r_max=0.1, filter="cone") for k in ks]
    b = PhotonMapBatch()
    pos, pw = (to_dev(np.concatenate([getattr(p, a) for p in ph]), cuda) for a in ("pos", "pow"))
    qp, qn = (to_dev(np.concatenate([getattr(x, a) for x in q]), cuda) for a in ("pos", "nrm"))
    b.build(pos, pw, poff)
    out = b.query(descs, qp, qn, qoff)
    lists = b.query(descs, qp, qn, qoff, want_nbr=True)
    torch.cuda.synchronize()
    at = 0
    for i, (n, m) in enumerate(sizes):
        if n and m:
            pm = PhotonMap(n, global_q_radius_max=0.1)
            pm.build(to_dev(ph[i].pos, cuda), to_dev(ph[i].pow, cuda))
            one = pm.query(to_dev(q[i].pos, cuda), to_dev(q[i].nrm, cuda), want_nbr=True, sorted_queries=False, **descs[i])
            s = slice(int(qoff[i]), int(qoff[i + 1]))
            for name in ("rad", "r2", "count"):
                for o in (out, lists):
                    assert torch.equal(o[name][s].view(torch.int32), one[name].view(torch.int32)), (i, name)
            assert torch.equal(lists["nbr"][at:at + m * ks[i]].view(m, ks[i]), one["nbr"]), i
        at += m * ks[i]


@pytest.mark.parametrize("nbr", [False, True])
def test_shared_walk_without_allocations(cuda, nbr):
    """pm_query_noalloc at its largest size shares walks too, and reads the queries
    through the order instead of from records."""
    n, nq, k = 60000, L.PM_NOALLOC_MAX_QUERIES, 40
    ph, q = gen.photons(n, seed=21, caustic_frac=0.2), gen.queries(nq, seed=22, cluster_frac=0.5)
    pm = PhotonMap(n, global_q_radius_max=0.1)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    qp, qn = to_dev(q.pos, cuda), to_dev(q.nrm, cuda)
    want = pm.query(qp, qn, want_nbr=nbr, sorted_queries=False, k=k, filter="cone")
    got = {name: torch.full_like(x, -1) for name, x in want.items()}
    d = pm.desc(k=k, filter="cone")
    lib = L.load()
    st = lib.pm_query_noalloc(pm.handle, C.byref(d), qp.data_ptr(), qn.data_ptr(), nq, got["rad"].data_ptr(),
                              got["nbr"].data_ptr() if nbr else None, got["r2"].data_ptr(), got["count"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
    assert st == L.PM_OK
    torch.cuda.synchronize()
    for name in want:
        assert torch.equal(got[name].view(torch.int32), want[name].view(torch.int32)), name


def test_shared_walk_from_two_threads(cuda):
    """Two maps queried by two host threads at once, with different k: handles are
    independent, every call answers every query."""
    n, nq = 20000, 262144
    ph, q = gen.photons(n, seed=31), gen.queries(nq, seed=32)
    arrays = [to_dev(a, cuda) for a in (ph.pos, ph.pow, q.pos, q.nrm)]
    work = []
    for k in (100, 128):
        pm = PhotonMap(n, global_q_radius_max=0.1)
        pm.build(*arrays[:2])
        want = pm.query(*arrays[2:], sorted_queries=False, k=k, filter="box")
        work.append((pm, k, want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    wrong = []

    def run(pm, k, want, stream):
        out = {name: torch.empty_like(x) for name, x in want.items()}
        for _ in range(50):
            with torch.cuda.stream(stream):
                for x in out.values():
                    x.fill_(-1)
                try:
                    pm.query(*arrays[2:], out=out, k=k, filter="box")
                except L.PMError as e:
                    wrong.append(str(e))
            stream.synchronize()
            wrong.extend(name for name in out if not torch.equal(out[name].view(torch.int32), want[name].view(torch.int32)))

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
