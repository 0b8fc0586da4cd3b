"""pm_build and pm_query recorded in a CUDA graph on storage reserved before:
replays on new inputs give the bits of direct calls.  The sizes take each kernel
that a capture may meet: the sorts of one cluster (up to 65,536), those of several
kernels, and the shared walk."""
import numpy as np
import pytest
import torch

from mnrt_b200 import gen
from mnrt_b200.photon_map import PhotonMap

pytestmark = pytest.mark.gpu


def to_dev(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


@pytest.mark.parametrize("n,nq", [(65536, 65536), (2, 3), (65537, 65537), (50000, 262144)])
def test_build_and_query_in_a_graph(cuda, n, nq):
    kw = dict(k=50, r_max=0.1, filter="cone")
    pm = PhotonMap(n, global_q_radius_max=0.1)
    pm.reserve(n, nq)
    ph, q = gen.photons(n, seed=1, caustic_frac=0.2), gen.queries(nq, seed=2)
    bufs = [to_dev(a, cuda) for a in (ph.pos, ph.pow, q.pos, q.nrm)]
    out = {name: torch.zeros(shape, dtype=dtype, device=cuda)
           for name, shape, dtype in (("rad", (nq, 4), torch.float32), ("r2", (nq,), torch.float32),
                                      ("count", (nq,), torch.int32), ("nbr", (nq, 50), torch.int32))}
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pm.build(*bufs[:2])
        pm.query(*bufs[2:], out=out, **kw)
    for seed in (3, 4):
        ph, q = gen.photons(n, seed=seed, caustic_frac=0.2), gen.queries(nq, seed=seed)
        for b, a in zip(bufs, (ph.pos, ph.pow, q.pos, q.nrm)):
            b.copy_(to_dev(a, cuda))
        for o in out.values():
            o.fill_(-1)
        graph.replay()
        direct = PhotonMap(n, global_q_radius_max=0.1)
        direct.build(*bufs[:2])
        want = direct.query(*bufs[2:], want_nbr=True, **kw)
        torch.cuda.synchronize()
        for name in out:
            assert torch.equal(out[name].view(torch.int32), want[name].view(torch.int32)), name
    del graph
