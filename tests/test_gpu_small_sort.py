"""Maps and query sets of up to 65,536 elements, which one cluster sorts: the
photons' tree order must be the stable order of their 39-bit Morton codes, and
every query must be answered once, at the edges of the blocks and clusters."""
import numpy as np
import pytest
import torch

from mnrt_b200 import gen
from mnrt_b200.photon_map import PhotonMap

pytestmark = pytest.mark.gpu


def to_dev(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def both(pm, qp, qn, **kw):
    """Outputs of the sorted and of the as-given query, which must agree bit for bit."""
    a = pm.query(qp, qn, want_nbr=True, **kw)
    b = pm.query(qp, qn, want_nbr=True, sorted_queries=False, **kw)
    torch.cuda.synchronize()
    for name in a:
        x, y = a[name].cpu().numpy(), b[name].cpu().numpy()
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), name


def morton39(p):
    lo, hi = p.min(0), p.max(0)
    ext = np.float32((hi - lo).max())
    scale = np.float32(65536.0) / ext if ext > 0 else np.float32(0)
    v = np.clip(((p - lo).astype(np.float32) * scale).astype(np.float32), 0, 65535).astype(np.uint64) >> np.uint64(3)
    code = np.zeros(len(p), np.uint64)
    for b in range(13):
        for a in range(3):
            code |= ((v[:, a] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + 2 - a)
    return code


@pytest.mark.parametrize("n", [2, 3, 31, 33, 1023, 1025, 2049, 16384, 16385, 32768, 32769, 65535, 65536, 65537])
@pytest.mark.parametrize("layout", ["packed", "reference"])
def test_small_map_order(cuda, n, layout):
    ph = gen.photons(n, seed=n, caustic_frac=0.2, layout=layout)
    ph.pos[n // 2:, :3] = ph.pos[: n - n // 2, :3]   # equal codes keep the caller's order
    pm = PhotonMap(n, global_q_radius_max=0.1)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda), packed=layout == "packed")
    _, pos, pw = pm.export_tree()
    order = pos[:, 3].view(np.uint32).astype(np.int64)
    assert np.array_equal(order, np.argsort(morton39(ph.pos[:, :3]), kind="stable"))
    assert np.array_equal(pos[:, :3], ph.pos[order, :3]) and np.array_equal(pw[:, :3], ph.pow[order, :3])
    info = pm.info()
    assert np.array_equal(np.array(info.bounds_min), ph.pos[:, :3].min(0))
    assert np.array_equal(np.array(info.bounds_max), ph.pos[:, :3].max(0))
    assert info.max_power == ph.pow[:, :3].max() and info.device_errors == 0


@pytest.mark.parametrize("nq", [2, 1023, 16385, 32769, 65536, 65537])
def test_small_query_sort(cuda, nq):
    """Every query answered once whatever sorts them."""
    ph = gen.photons(2000, seed=1, caustic_frac=0.2)
    q = gen.queries(nq, seed=2, cluster_frac=0.5)
    pm = PhotonMap(2000, global_q_radius_max=0.2)
    pm.build(to_dev(ph.pos, cuda), to_dev(ph.pow, cuda))
    both(pm, to_dev(q.pos, cuda), to_dev(q.nrm, cuda), k=10, r_max=0.2, filter="box")
