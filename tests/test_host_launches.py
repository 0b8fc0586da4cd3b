"""The engine's host code without a GPU: its sources linked with a CUDA runtime
that keeps a log instead of launching (tests/cpp/host_runtime.cpp).  Shows what
a call asks the runtime for, and what it does when the runtime refuses."""
import ctypes as C
import shutil
import subprocess
import threading
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import pytest

from mnrt_b200 import _lib as L
from mnrt_b200 import build

HERE = Path(__file__).resolve().parent


class Engine:
    """The host-only library: handles, calls and the runtime's log."""

    def __init__(self, path):
        self.lib = L.load(path)
        self.lib.host_log.restype = C.c_char_p
        self.lib.host_set.argtypes = [C.c_char_p, C.c_int]

    def log(self):
        return self.lib.host_log().decode().splitlines()

    def set(self, name, value):
        self.lib.host_set(name.encode(), value)

    def map(self, n, nq=0):
        h = C.c_void_p()
        assert self.lib.pm_create(C.byref(h), 0, None, None, 0.1) == L.PM_OK
        assert self.lib.pm_reserve(h, n, nq) == L.PM_OK
        return h

    def build(self, h, n):   # the photon arrays are never read: nothing is launched
        return self.lib.pm_build(h, 16, 32, n, L.PM_PHOTONS_PACKED, None)

    def query(self, h, nq, call="pm_query", lists=False, **kw):
        return getattr(self.lib, call)(h, C.byref(desc(**kw)), 16, 32, nq, 48, 64 if lists else None, None, None, None)


def desc(**kw):
    return L.QueryDesc(**{**dict(k=50, r_max=0.1, filter=L.PM_FILTER_CONE, cone_k=1.0, mode=L.PM_MODE_EXACT, min_found=0,
                                 order=L.PM_ORDER_SORTED, refine_iters=2), **kw})


def launched(log, name):
    return [x for x in log if x.startswith(("launch " + name, "cluster " + name))]


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("host")

    def compile(src):   # PTX only: nothing of it runs
        out = tmp / (src + ".o")
        cmd = [build.nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-w", "-std=c++17",
               "--expt-relaxed-constexpr", "-cudart", "none", "-Xcompiler", "-fPIC,-fvisibility=hidden", "-I",
               str(build.ROOT / "include"), "-c", str(build.CSRC / src), "-o", str(out)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        return str(out)

    with ThreadPoolExecutor(8) as pool:
        objects = list(pool.map(compile, build.SOURCES))
    lib = tmp / "libpmgpu_host.so"
    cuda = Path(shutil.which("nvcc") or build.nvcc()).resolve().parent.parent
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-fvisibility=hidden", "-I", str(cuda / "include"),
                        str(HERE / "cpp" / "host_runtime.cpp"), *objects, "-Wl,--no-undefined", "-o", str(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return Engine(lib)


@pytest.mark.parametrize("call,kernel", [("pm_query", "k_knn_shared"), ("pm_query_bruteforce", "k_knn_brute")])
def test_shared_memory_limit_is_never_lowered(engine, call, kernel):
    """A kernel's limit on dynamic shared memory belongs to the process: a call
    that lowers it, even for a moment, fails the launches of other threads."""
    n, nq = 1000, 262144
    handles = [engine.map(n, nq) for _ in range(2)]
    for h in handles:
        assert engine.build(h, n) == L.PM_OK
    engine.log()
    status = []

    def work(h, k):
        for _ in range(200):
            status.append(engine.query(h, nq, call, k=k))

    threads = [threading.Thread(target=work, args=(h, k)) for h, k in zip(handles, (100, 128))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    log = engine.log()
    assert launched(log, kernel)
    assert not [x for x in log if x.startswith(("lowered", "refused"))]
    assert set(status) == {L.PM_OK}
    for h in handles:
        engine.lib.pm_destroy(h)


@pytest.mark.parametrize("lists", [False, True])
def test_shared_walk_asks_for_its_block_size_once(engine, lists):
    n, nq = 3000, 262144
    h = engine.map(n, nq)
    assert engine.build(h, n) == L.PM_OK
    asked = []
    for k in (100, 100, 128, 100, 128):
        engine.log()
        assert engine.query(h, nq, lists=lists, k=k) == L.PM_OK
        log = engine.log()
        assert len(launched(log, "k_knn_shared")) == 1
        asked.append(sum(x.startswith("occupancy k_knn_shared") for x in log))
    assert asked == [5, 0, 5, 0, 0]
    engine.lib.pm_destroy(h)


@pytest.mark.parametrize("setting,value", [("clusters", 0), ("refuse_clusters", 1)])
@pytest.mark.parametrize("n", [2, 16385, 32769, 65536])
def test_small_sorts_without_room_for_a_cluster(engine, setting, value, n):
    """Maps and query sets of up to 65,536 elements take the sorts of several
    kernels where one cluster does not fit, or its launch is refused."""
    several = ["k_bounds", "k_morton", "k_digit_scatter<unsigned long", "k_query_order", "k_digit_scatter<unsigned int"]
    try:
        for fits in (True, False):
            h = engine.map(n, n)
            engine.set(setting, value if not fits else {"clusters": 8, "refuse_clusters": 0}[setting])
            engine.log()
            assert engine.build(h, n) == L.PM_OK and engine.query(h, n) == L.PM_OK
            log = engine.log()
            assert len(launched(log, "k_small_build")) == len(launched(log, "k_small_query_sort")) == (1 if fits else 0)
            assert [bool(launched(log, x)) for x in several] == [not fits] * len(several)
            assert launched(log, "k_knn_group")
            assert engine.build(h, n) == L.PM_OK and engine.query(h, n) == L.PM_OK   # asked once, answered alike
            again = engine.log()
            assert not [x for x in again if x.startswith("clusters ")] and [x for x in log if x.startswith("clusters ")]
            assert bool(launched(again, "k_small_build")) == bool(launched(again, "k_small_query_sort")) == fits
            engine.lib.pm_destroy(h)
    finally:
        engine.set("clusters", 8)
        engine.set("refuse_clusters", 0)


@pytest.mark.parametrize("nq,shared", [(262143, False), (262144, True)])
def test_batch_lays_records_out_for_the_shared_walk_only(engine, nq, shared):
    b = C.c_void_p()
    assert engine.lib.pm_batch_create(C.byref(b)) == L.PM_OK
    photons, queries = (C.c_uint32 * 3)(0, 400, 5000), (C.c_uint32 * 3)(0, 7, nq)
    descs = (L.QueryDesc * 2)(desc(), desc())
    assert engine.lib.pm_batch_build(b, 16, 32, photons, 2, L.PM_PHOTONS_PACKED, None) == L.PM_OK
    engine.log()
    assert engine.lib.pm_batch_query(b, descs, 16, 32, queries, 48, None, None, None, None) == L.PM_OK
    log = engine.log()
    assert len(launched(log, "k_knn_shared<true")) == len(launched(log, "k_gather_queries")) == int(shared)
    assert len(launched(log, "k_knn_group<32, false, true, true>")) == int(not shared)
    assert engine.lib.pm_batch_destroy(b) == L.PM_OK


@pytest.mark.parametrize("nq,k,records", [(1, 8, False), (15999, 2, False), (16000, 2, True), (300, 128, True)])
def test_adjoint_lays_photon_records_out_for_many_pairs_only(engine, nq, k, records):
    """The records cost every photon: below 32 pairs a photon the adjoint gathers
    through the inverse permutation."""
    n = 1000
    h = engine.map(n, nq)
    assert engine.build(h, n) == L.PM_OK
    engine.log()
    assert engine.lib.pm_query_backward(h, C.byref(desc(k=k)), 16, 32, nq, 48, 64, None, 80, 96, 112, None) == L.PM_OK
    log = engine.log()
    assert len(launched(log, "k_bwd_pack")) == len(launched(log, "k_bwd_prep<true, true>")) == int(records)
    assert len(launched(log, "k_bwd_prep<true, false>")) == int(not records)
    engine.lib.pm_destroy(h)


@pytest.mark.parametrize("n,wide", [(39999, False), (40000, True)])
def test_adjoint_reduces_few_photons_by_short_loads(engine, n, wide):
    h = engine.map(n, 100)
    assert engine.build(h, n) == L.PM_OK
    engine.log()
    assert engine.lib.pm_query_backward(h, C.byref(desc(k=8)), 16, 32, 100, 48, 64, None, 80, 96, 112, None) == L.PM_OK
    assert len(launched(engine.log(), f"k_bwd_reduce<{str(wide).lower()}>")) == 1
    engine.lib.pm_destroy(h)


def test_first_adjoint_takes_no_storage_for_photon_records(engine):
    """The adjoint's 32-byte photon records lie in the build's scratch, which is idle
    between builds: a map's first adjoint allocates four bytes a photon an array."""
    n, nq = 100000, 10
    h = engine.map(n, nq)
    assert engine.build(h, n) == L.PM_OK
    engine.log()
    assert engine.lib.pm_query_backward(h, C.byref(desc(k=1)), 16, 32, nq, 48, 64, None, 80, 96, 112, None) == L.PM_OK
    log = engine.log()
    sizes = [int(x.split()[1]) for x in log if x.startswith("malloc")]
    assert len(sizes) == 6 and max(sizes) <= 4 * (n + 1)
    assert launched(log, "k_bwd_prep")
    engine.lib.pm_destroy(h)


@pytest.mark.parametrize("n,nq,k,lists,shared", [
    (1048576, 2073600, 100, False, True), (4194304, 8388608, 64, False, True), (1048576, 1048576, 64, True, True),
    (250007, 400009, 100, True, True), (3000, 262144, 100, False, True), (3000, 262143, 100, False, False),
    # sets that were faster one by one: few queries a photon for their k, nearly every photon in every list
    (1048576, 655360, 128, False, False), (4000000, 1280000, 100, False, False), (600000, 495742, 128, False, False),
    (65536, 262144, 1, False, False), (1048576, 655360, 1, False, False), (4000000, 2560000, 1, False, False),
    (100, 524288, 100, True, False), (100, 524288, 50, True, False), (100, 524288, 100, False, True),
])
def test_which_queries_share_walks(engine, n, nq, k, lists, shared):
    h = engine.map(n, nq)
    assert engine.build(h, n) == L.PM_OK
    engine.log()
    assert engine.query(h, nq, lists=lists, k=k) == L.PM_OK
    assert bool(launched(engine.log(), "k_knn_shared")) == shared
    assert engine.lib.pm_query_kernel(h) == (b"k_knn_shared" if shared else b"k_knn_group")
    engine.lib.pm_destroy(h)


@pytest.mark.parametrize("maps,shared", [
    # (photons, queries, k) of each map: dense, sparse, and both; tiny maps count neither way
    ([(50000, 200000, 64)] * 3, True), ([(300000, 30000, 64)] * 20, False), ([(300000, 400000, 64), (300000, 30000, 64)], True),
    ([(300000, 300000, 64)] + [(300000, 60000, 64)] * 10, False), ([(300, 480, 8)] * 3000, False),
    ([(300, 480, 8)] * 1000 + [(50000, 200000, 64)] * 2, True),
])
def test_which_batches_share_walks(engine, maps, shared):
    b = C.c_void_p()
    assert engine.lib.pm_batch_create(C.byref(b)) == L.PM_OK
    off = lambda i: (C.c_uint32 * (len(maps) + 1))(*[sum(m[i] for m in maps[:j]) for j in range(len(maps) + 1)])
    photons, queries = off(0), off(1)
    descs = (L.QueryDesc * len(maps))(*[desc(k=m[2]) for m in maps])
    assert engine.lib.pm_batch_build(b, 16, 32, photons, len(maps), L.PM_PHOTONS_PACKED, None) == L.PM_OK
    engine.log()
    assert engine.lib.pm_batch_query(b, descs, 16, 32, queries, 48, None, None, None, None) == L.PM_OK
    assert bool(launched(engine.log(), "k_knn_shared<true")) == shared
    assert engine.lib.pm_batch_destroy(b) == L.PM_OK


@pytest.mark.parametrize("n,nq,kernels", [
    (64, 16383, ["k_compat_query<false>"]), (64, 16384, ["k_compat_start"]),
    (65, 65535, ["k_compat_query<false>"]), (65, 65536, ["k_compat_start", "k_compat_query<true>"]),
])
def test_many_small_ranges_are_answered_by_threads(engine, n, nq, kernels):
    """A warp for each of many queries with a photon or two in range took up to 26 times a
    thread's share of the chip."""
    h = engine.map(n, nq)
    assert engine.build(h, n) == L.PM_OK
    engine.log()
    assert engine.query(h, nq, mode=L.PM_MODE_ZHOU_COMPAT) == L.PM_OK
    assert [x.split(" grid")[0].split(" ", 1)[1] for x in engine.log() if " k_compat_" in x][1:] == kernels   # after the nodes
    engine.lib.pm_destroy(h)


def test_autotuners_time_a_shared_walk_once_per_leaf_and_rounds(engine):
    """A shared walk chooses its own warps per block: timing it for each setting would
    pick among equals by noise, and leave searches one by one with that setting."""
    n, nq = 3000, 262144
    q = np.zeros((nq + 1, 4), np.float32)
    ptr = q.ctypes.data + (-q.ctypes.data) % 16
    best = L.Tuning()
    h = engine.map(n, nq)
    engine.log()
    assert engine.lib.pm_autotune(h, 16, 32, n, L.PM_PHOTONS_PACKED, C.byref(desc(k=100)), ptr, ptr, nq, 0, C.byref(best),
                                  None) == L.PM_OK
    log = engine.log()
    assert len(launched(log, "k_knn_shared<false, false>")) == 2 * 5 * 2   # each is timed the second time
    assert all(" block 128 " in x for x in launched(log, "k_knn_group<32, true, false, true>"))
    assert len(launched(log, "k_knn_group<32, false, false, false>")) == 2 * 5 * 3 * 2
    engine.lib.pm_destroy(h)

    b = C.c_void_p()
    assert engine.lib.pm_batch_create(C.byref(b)) == L.PM_OK
    photons, queries, descs = (C.c_uint32 * 2)(0, n), (C.c_uint32 * 2)(0, nq), (L.QueryDesc * 1)(desc(k=100))
    assert engine.lib.pm_batch_autotune(b, 16, 32, photons, 1, L.PM_PHOTONS_PACKED, descs, 48, 64, queries, 80,
                                        C.byref(best), None) == L.PM_OK
    log = engine.log()
    assert len(launched(log, "k_knn_shared<true, false>")) == 2 * 5 * 2
    assert all(" block 128 " in x for x in launched(log, "k_knn_group<32, true, true, true>"))
    assert engine.lib.pm_batch_destroy(b) == L.PM_OK


@pytest.mark.parametrize("nq,layout,qpw,order,blocks", [
    # 148 SMs of 8 blocks of 4 warps: a chunk of 14 rounds keeps 65,536 queries to one for each of 4,736 warps
    (65536, L.PM_KBUF_WIDE, 1, L.PM_ORDER_AS_GIVEN, 1171), (65536, L.PM_KBUF_WIDE, 1, L.PM_ORDER_SORTED, 1171),
    (16384, L.PM_KBUF_WIDE, 1, L.PM_ORDER_AS_GIVEN, 1024),       # 4 rounds, 4,096 warps
    (16384, L.PM_KBUF_WIDE, 1, L.PM_ORDER_SORTED, 1184),         # 3 rounds, 5,462 chunks
    (4095, L.PM_KBUF_WIDE, 1, L.PM_ORDER_SORTED, 1024),          # a round each
])
def test_chunks_of_small_launches(engine, nq, layout, qpw, order, blocks):
    n = 1000
    h = engine.map(n, nq)
    assert engine.lib.pm_set_tuning(h, 32, 4, 32, qpw, layout) == L.PM_OK
    assert engine.build(h, n) == L.PM_OK
    engine.log()
    assert engine.query(h, nq, order=order) == L.PM_OK
    (line,) = [x for x in engine.log() if "k_knn_group<32, false, false" in x and x.startswith("launch")]
    assert f" grid {blocks} block 128 " in line
    engine.lib.pm_destroy(h)
