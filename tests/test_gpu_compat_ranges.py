"""PM_MODE_ZHOU_COMPAT bit for bit against the oracle where the warp's range
search can go wrong: a single photon, ranges that hold more photons than the
kernel keeps for its second pass, leaves counted as a whole, query counts beside
a block's."""
import numpy as np
import pytest
import torch

from mnrt_b200 import _lib as L
from mnrt_b200 import gen
from mnrt_b200.photon_map import PhotonMap
from tests.test_gpu_parity import format_errors, radiance_errors

pytestmark = pytest.mark.gpu


def to_dev(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


@pytest.mark.parametrize("n,nq,k,r,iters,filt", [
    (1, 40, 3, 0.2, 2, "box"),
    (700, 1025, 128, 0.5, 0, "cone"),            # no refinement: ranges beyond the kept photons
    (30000, 3001, 20, 0.3, 1, "epanechnikov"),   # node estimates; bins counted a leaf at a time
    (30000, 999, 128, 0.1, 5, "cone"),
])
def test_compat_ranges(cuda, oracle_mod, n, nq, k, r, iters, filt):
    ph = gen.photons(n, seed=n, caustic_frac=0.5)
    q = gen.queries(nq, seed=nq, cluster_frac=0.5)
    pm = PhotonMap(n, global_q_radius_max=r, knn_target_count=k)
    pm.set_tuning(leaf_size=16)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    qp, qn = to_dev(q.pos, cuda), to_dev(q.nrm, cuda)
    out = pm.query(qp, qn, mode=L.PM_MODE_ZHOU_COMPAT, refine_iters=iters, filter=filt, min_found=8)
    radii = pm.compute_query_radii(qp, refine_iters=iters)
    torch.cuda.synchronize()
    nodes, tpos, tpow = pm.export_tree()
    o_radius, o_count, o_r2, o_rad = oracle_mod.compat(nodes, tpos, tpow, q.pos, q.nrm, k, r, iters, filt, 1.0, 8)
    assert np.array_equal(radii.cpu().numpy(), o_radius)
    assert np.array_equal(out["count"].cpu().numpy().view(np.uint32), o_count)
    assert np.array_equal(out["r2"].cpu().numpy(), o_r2)
    e = radiance_errors(out["rad"].cpu().numpy()[:, :3], o_rad)
    assert e["max"] <= 1e-5, format_errors(e)
    assert pm.info().device_errors == 0


@pytest.mark.parametrize("leaf", [32, 64])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_compat_counts_finite_photons_only(cuda, leaf, bad):
    """Photons without a finite position are in no range: radii, counts and r^2 are
    those of the map of the other photons (a tree too small for node estimates,
    so that a radius depends on the photons in range alone)."""
    n, nq, kw = 4000, 2000, dict(k=50, r_max=0.6)
    ph = gen.photons(n, seed=5, caustic_frac=0.5)
    q = gen.queries(nq, seed=6)
    good = np.arange(n) % 7 != 3
    ph.pos[~good, 0] = bad
    qp, qn = to_dev(q.pos, cuda), to_dev(q.nrm, cuda)
    got = []
    for keep in (np.ones(n, bool), good):
        pm = PhotonMap(n, global_q_radius_max=0.6)
        pm.set_tuning(leaf_size=leaf)
        pm.build(to_dev(ph.pos[keep], cuda), to_dev(ph.pow[keep], cuda))
        pm.clear_errors()   # the header's error bits may be cleared at any time
        out = pm.query(qp, qn, mode=L.PM_MODE_ZHOU_COMPAT, filter="box", **kw)
        got.append([pm.compute_query_radii(qp, **kw), out["count"], out["r2"]])
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n,leaf,k,r,iters,filt", [
    (64, 1, 20, 0.3, 2, "cone"),              # a map that a thread answers whole
    (65, 64, 20, 0.3, 2, "cone"),             # one photon more: by ranges
    (1500, 32, 20, 0.02, 2, "box"),           # ranges of a leaf or two
    (1500, 32, 3, 0.05, 0, "epanechnikov"),   # beside those that a warp takes
    (20000, 32, 50, 0.003, 2, "box"),         # ranges of no photon
])
def test_compat_small_ranges_of_many_queries(cuda, oracle_mod, n, leaf, k, r, iters, filt):
    """From 65,536 queries up (16,384 on a map of 64 photons) a thread answers a query
    whose range is a leaf or two, and a warp the others."""
    nq = 16384 if n <= 64 else 65537
    ph = gen.photons(n, seed=n, caustic_frac=0.3)
    q = gen.queries(nq, seed=nq, cluster_frac=0.5)
    q.pos[7, 1] = np.inf
    pm = PhotonMap(n, global_q_radius_max=r, knn_target_count=k)
    pm.set_tuning(leaf_size=leaf)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    qp, qn = to_dev(q.pos, cuda), to_dev(q.nrm, cuda)
    out = pm.query(qp, qn, mode=L.PM_MODE_ZHOU_COMPAT, refine_iters=iters, filter=filt, min_found=2)
    radii = pm.compute_query_radii(qp, refine_iters=iters)
    few = pm.compute_query_radii(qp[:500], refine_iters=iters)   # a warp each
    torch.cuda.synchronize()
    assert pm.info().device_errors == L.PM_DEVERR_QNONFINITE
    assert torch.equal(radii[:500], few)
    assert float(radii[7]) == np.float32(r) and int(out["count"][7]) == 0 and not out["rad"][7].any()
    fin = np.isfinite(q.pos[:, :3]).all(1)
    nodes, tpos, tpow = pm.export_tree()
    o_radius, o_count, o_r2, o_rad = oracle_mod.compat(nodes, tpos, tpow, q.pos[fin], q.nrm[fin], k, r, iters, filt, 1.0, 2)
    assert np.array_equal(radii.cpu().numpy()[fin], o_radius)
    assert np.array_equal(out["count"].cpu().numpy().view(np.uint32)[fin], o_count)
    assert np.array_equal(out["r2"].cpu().numpy()[fin], o_r2)
    # 1e-5 of FP64, and the fixed point's resolution: a term is rounded to the largest flux / 2^40 (estimates
    # of two photons at the edge of their range, weight 1e-8, come near it)
    rad = out["rad"].cpu().numpy()[fin, :3].astype(np.float64)
    step = o_count * pm.info().max_power * 2.0 ** -41 * 2 / (np.pi * np.maximum(o_r2, 1e-30))
    assert (np.abs(rad - o_rad) <= 1e-5 * np.abs(o_rad) + step[:, None]).all()
