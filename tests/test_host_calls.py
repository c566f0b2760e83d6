"""CPU tests of the library's host side against a fake CUDA runtime (tests/cpp/fake_cudart.cpp, linked with the
library's own objects): which kernels a call launches, what it does under stream capture, and what it leaves behind when
an allocation fails. Kernels do nothing there, so results are not looked at; the GPU tests check those."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

OPT_TC_KERNEL, OPT_LOOP_MODE, OPT_ITEM_WORK = 1, 2, 4
GA_ERR_CUDA, GA_ERR_OUT_OF_MEMORY = 3, 4


class Lib:
    """The library over the fake runtime."""

    def __init__(self, path):
        self.c = C.CDLL(path)
        self.c.fake_log.restype = C.c_char_p
        self.c.fake_live.restype = C.c_longlong
        self.c.fake_fail_in.argtypes = [C.c_longlong]

    def __getattr__(self, name):
        return getattr(self.c, name)

    def leaked(self):
        return self.c.fake_live() - self.before

    def log(self):
        return self.c.fake_log().decode().splitlines()

    def launches(self):
        return [line.split()[1] for line in self.log() if line.startswith("launch")]

    def graph(self, n=64, stream=None):
        """A handle of a path of n vertices (n - 1 edges)."""
        rowptr = np.minimum(np.arange(n + 1, dtype=np.uint32), n - 1)
        col = np.arange(1, n, dtype=np.uint32)
        h = C.c_void_p()
        s = self.c.ga_graph_create(rowptr.ctypes.data_as(C.c_void_p), col.ctypes.data_as(C.c_void_p), n, n - 1, 0, stream,
                                   C.byref(h))
        return s, h


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    from graph_analyzer_b200 import build
    os.makedirs(build.BUILD_DIR, exist_ok=True)
    objs = [build._compile(s, False) for s in build._sources()]
    out = str(tmp_path_factory.mktemp("fake") / "libga_fake.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-fopenmp", "-Wl,-Bsymbolic", "-I", cuda,
                           *objs, os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", out, "-lpthread"])
    return Lib(out)


@pytest.fixture
def lib(fake_lib):
    fake_lib.fake_reset()
    fake_lib.before = fake_lib.fake_live()
    yield fake_lib
    fake_lib.fake_reset()


@pytest.mark.parametrize("shard", [False, True])
@pytest.mark.parametrize("kernel", [1, 2])
def test_enqueued_counts_share_no_counters(lib, kernel, shard):
    """An _async count clears the caller's total (and, in the hash form, work queues that are its own) before its kernel:
    passes enqueued on one handle by several captures then share nothing they write."""
    s, g = lib.graph()
    assert s == 0 and lib.ga_graph_set_option(g, OPT_TC_KERNEL, C.c_int64(kernel)) == 0 and lib.ga_graph_prepare(g) == 0
    stream = C.c_void_p(0x1000)
    assert lib.ga_graph_set_stream(g, stream) == 0
    totals = (C.c_uint64 * 2)(7, 7)
    cleared = []
    for i in range(2):
        lib.fake_reset()
        lib.fake_capture(stream, 1)
        at = C.addressof(totals) + 8 * i
        if shard:
            assert lib.ga_tc_count_shard_async(g, 1, 3, C.c_void_p(at)) == 0
        else:
            assert lib.ga_tc_count_async(g, C.c_void_p(at)) == 0
        lib.fake_capture(stream, 0)
        log = [line for line in lib.log() if line.endswith("captured")]
        memsets = [line.split()[1:3] for line in log if line.startswith("memset")]
        assert [str(at), "8"] in memsets
        assert any(line.startswith("launch") for line in log[log.index(f"memset {at} 8 captured"):])
        cleared.append({m[0] for m in memsets})
        assert len(cleared[i]) == kernel          # the total, and the hash form's queues
    assert not cleared[0] & cleared[1]
    assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0


def captured_call(lib, g, call):
    """(status, log) of call(handle) on a handle whose stream is being captured."""
    stream = C.c_void_p(0x2000)
    assert lib.ga_graph_set_stream(g, stream) == 0
    lib.fake_reset()
    lib.fake_capture(stream, 1)
    s = call(g)
    log = lib.log()
    lib.fake_capture(stream, 0)
    return s, log


TOTAL = C.c_uint64(0)
CALLS = {
    "async": lambda lib, g: lib.ga_tc_count_async(g, C.byref(TOTAL)),
    "shard_async": lambda lib, g: lib.ga_tc_count_shard_async(g, 0, 2, C.byref(TOTAL)),
    "count": lambda lib, g: lib.ga_tc_count(g, C.byref(TOTAL)),
    "shard": lambda lib, g: lib.ga_tc_count_shard(g, 0, 2, C.byref(TOTAL)),
    "prepare": lambda lib, g: lib.ga_graph_prepare(g),
    "cores": lambda lib, g: lib.ga_core_decomposition(g, None, C.byref((C.c_uint32 * 2)())),
    "peel": lambda lib, g: lib.ga_batch_peel(g, C.c_uint64(1), C.c_uint64(10), C.byref((C.c_uint64 * 3)()), None),
}


@pytest.mark.parametrize("call", list(CALLS))
def test_nothing_is_built_inside_a_capture(lib, call):
    """On a handle that nothing has prepared, a call under stream capture is refused and leaves nothing in the capture:
    an index recorded there would not exist until the graph runs. The same call afterwards builds what it needs."""
    s, g = lib.graph(n=200)
    assert s == 0 and lib.ga_graph_set_option(g, OPT_TC_KERNEL, C.c_int64(2)) == 0
    s, log = captured_call(lib, g, lambda g: CALLS[call](lib, g))
    assert s == GA_ERR_CUDA and not [line for line in log if line.endswith("captured")]
    lib.fake_reset()
    assert CALLS[call](lib, g) == 0 and any("k_in_lists" in k for k in lib.launches())
    assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0


@pytest.mark.parametrize("call", ["cores", "peel"])
def test_no_loop_state_is_built_inside_a_capture(lib, call):
    s, g = lib.graph(n=200)
    assert s == 0 and lib.ga_graph_prepare(g) == 0
    for run_other_first in (False, True):
        if run_other_first:   # the other loop's state stands, this one's may not
            assert CALLS["peel" if call == "cores" else "cores"](lib, g) == 0
        s, log = captured_call(lib, g, lambda g: CALLS[call](lib, g))
        assert s == GA_ERR_CUDA and not [line for line in log if line.startswith("alloc") and line.endswith("captured")]
    assert CALLS[call](lib, g) == 0
    assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0


@pytest.mark.parametrize("call,kernel", [("async", "k_tc_octs"), ("shard_async", "k_tc_hash")])
@pytest.mark.parametrize("before", ["prepare", "count", "async"])
def test_capture_after_a_first_call(lib, before, call, kernel):
    """After ga_graph_prepare, a synchronous count (which may have done without the index) or an enqueued one, counts and
    shards can be captured: what they still need is built outside the capture, and the kernel is the handle's choice."""
    n = 300                                      # one signature: the first handle tunes (one-thread form), later ones know
    s, first = lib.graph(n=n)
    assert s == 0 and lib.ga_graph_prepare(first) == 0
    s, g = lib.graph(n=n)
    assert s == 0
    lib.fake_reset()
    assert CALLS[before](lib, g) == 0
    if before == "count":
        assert [k for k in lib.launches() if "k_tc_" in k] and not any("k_in_lists" in k for k in lib.launches())
    if before == "async":                        # (enqueued on a handle whose choice nothing has looked up: the hash form)
        kernel = "k_tc_hash"
    s, log = captured_call(lib, g, lambda g: CALLS[call](lib, g))
    assert s == 0
    inside = [line for line in log if line.endswith("captured")]
    assert not [line for line in inside if line.startswith(("alloc", "sync", "record", "wait"))]
    ran = [line for line in inside if line.startswith("launch")]
    assert kernel in ran[-1] and all("k_tc_" in k or "k_shard_bounds" in k for k in ran)
    for h in (first, g):
        assert lib.ga_graph_destroy(h) == 0
    assert lib.leaked() == 0


def test_captured_passes_keep_their_work_lists(lib):
    """Work lists that a captured pass reads stay as they are when other options, or the autotuner, make new ones."""
    s, g = lib.graph()
    assert s == 0 and lib.ga_graph_set_option(g, OPT_TC_KERNEL, C.c_int64(2)) == 0 and lib.ga_graph_prepare(g) == 0
    for captured in (False, True, False):
        if captured:
            assert captured_call(lib, g, lambda g: CALLS["async"](lib, g))[0] == 0
        held = lib.leaked()
        assert lib.ga_graph_set_option(g, OPT_ITEM_WORK, C.c_int64(16 + 16 * captured + held)) == 0
        assert lib.ga_graph_prepare(g) == 0
        assert lib.leaked() == held + (4 if captured else 0)    # anchors, first and last in-edges, the bins' sizes
    assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0


@pytest.mark.parametrize("mode,graph", [(0, False), (2, True)])
def test_core_loop_honours_the_loop_mode(lib, mode, graph):
    """A core loop that fits one cluster is launched round by round only when the mode is automatic; mode 2 is one launch of
    a captured graph, without a synchronisation inside the loop."""
    s, g = lib.graph(n=200)
    assert s == 0 and lib.ga_graph_set_option(g, OPT_LOOP_MODE, C.c_int64(mode)) == 0 and lib.ga_graph_prepare(g) == 0
    for _ in range(2):
        lib.fake_reset()
        assert CALLS["cores"](lib, g) == 0
        log = lib.log()
        direct = [line for line in log if "k_core_small_rounds" in line and not line.endswith("captured")]
        assert (log.count("graph launch"), len(direct)) == ((1, 0) if graph else (0, 1))
    assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0


def test_prepare_returns_when_the_index_stands(lib):
    """ga_graph_prepare waits for what it built - also where it need not time candidates, because the signature is known -
    and for nothing when nothing was missing (it may then be called under capture)."""
    n = 400
    handles = [lib.graph(n=n) for _ in range(2)]
    assert all(s == 0 for s, _ in handles)
    for _, g in handles:
        lib.fake_reset()
        assert lib.ga_graph_prepare(g) == 0
        log = lib.log()
        launches = [i for i, line in enumerate(log) if line.startswith("launch")]
        assert launches and "sync" in log[launches[-1]:]
        s, log = captured_call(lib, g, lambda g: CALLS["prepare"](lib, g))
        assert s == 0 and not log
    for _, g in handles:
        assert lib.ga_graph_destroy(g) == 0
    assert lib.leaked() == 0


WORDS = (C.c_uint64 * 5000)()
CALLS.update({
    "supports": lambda lib, g: lib.ga_tc_support_edges(g, WORDS, None),
    "vertex_supports": lambda lib, g: lib.ga_tc_support_vertices(g, WORDS, None),
    "participation": lambda lib, g: lib.ga_tc_participation(g, WORDS, WORDS, None),
    "density": lambda lib, g: lib.ga_core_level_density(g, WORDS, 0, C.byref(TOTAL), C.byref(TOTAL)),
    "exact": lambda lib, g: lib.ga_exact_densest(g, C.byref((C.c_uint64 * 4)()), None),
    "lists_then_peel": lambda lib, g: CALLS["exact"](lib, g) or CALLS["peel"](lib, g),
})


def check_after_failed_allocations(lib, call, setup=()):
    """Lets the k-th allocation of `call` fail, for every k: the call reports it or does without; a repeat succeeds and leaves
    the handle with as many blocks as one that was never disturbed; destroying the handle frees everything."""
    held = None
    for k in range(-1, 200):
        s, g = lib.graph(n=5000)                  # (scans of more than one tile allocate too)
        assert s == 0 and lib.ga_graph_set_option(g, OPT_TC_KERNEL, C.c_int64(2)) == 0
        for c in setup:
            assert CALLS[c](lib, g) == 0
        before = lib.leaked()
        lib.fake_fail_in(C.c_longlong(k))
        s = CALLS[call](lib, g)
        failed = lib.fake_failed()
        lib.fake_fail_in(C.c_longlong(-1))
        assert s in (0, GA_ERR_OUT_OF_MEMORY) and (failed or s == 0), (k, s)
        if s:
            assert CALLS[call](lib, g) == 0, k
        if k < 0:
            held = lib.leaked() - before
        elif s:
            assert lib.leaked() - before == held, k
        assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0, k
        if k >= 0 and not failed:
            return k
    raise AssertionError("still allocating")


@pytest.mark.parametrize("call,setup", [("prepare", ()), ("count", ()), ("supports", ()), ("vertex_supports", ()),
                                        ("participation", ()), ("density", ()), ("shard", ("prepare",)), ("shard", ())])
def test_calls_after_failed_allocations(lib, call, setup):
    assert check_after_failed_allocations(lib, call, setup) > 0


def test_shard_cut_after_a_failed_allocation(lib):
    """A work prefix whose scan could not run is not kept: the next call makes it again."""
    for k in (0, 1):                             # the prefix itself, the scan's temporary
        s, g = lib.graph(n=5000)
        assert s == 0 and CALLS["prepare"](lib, g) == 0
        lib.fake_fail_in(C.c_longlong(k))
        assert CALLS["shard"](lib, g) == GA_ERR_OUT_OF_MEMORY and lib.fake_failed()
        lib.fake_reset()
        assert CALLS["shard"](lib, g) == 0 and any("k_scan_tiles" in name for name in lib.launches())
        assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0


@pytest.mark.parametrize("call", ["peel", "cores", "exact", "lists_then_peel"])
def test_loops_after_failed_allocations(lib, call):
    """Loop state and incidence lists of which an allocation failed are not taken for complete ones by the next call."""
    assert check_after_failed_allocations(lib, call, ("prepare",)) > 0


class ServerConfig(C.Structure):
    _fields_ = [("device", C.c_int), ("budget", C.c_uint64), ("slots", C.c_uint32), ("fold_max_graphs", C.c_uint32),
                ("fold_max_edges", C.c_uint32), ("small_slots", C.c_uint32), ("pin_min_edges", C.c_uint32)]


class RequestResult(C.Structure):
    _fields_ = [("status", C.c_int), ("triangles", C.c_uint64), ("peel", C.c_uint64 * 3), ("core", C.c_uint32 * 2),
                ("queue_ms", C.c_double), ("run_ms", C.c_double), ("folded", C.c_uint32), ("resident_hit", C.c_uint32)]


class ServerStats(C.Structure):
    _fields_ = [(f, C.c_uint64) for f in ("submitted", "completed", "folded", "evictions", "resident", "resident_bytes",
                                          "peak_reserved", "queued", "running", "reserved")]


def serve_counts(lib, sizes, requests, budget):
    """Counts, one after the other, of paths of sizes[i] vertices on a server of one worker: the results and the final
    statistics."""
    cfg = ServerConfig(0, budget, 1, 1, 1, 0xFFFFFFFF, 0)
    s = C.c_void_p()
    assert lib.ga_server_create(C.byref(cfg), C.byref(s)) == 0
    ids, results = [], []
    for n in sizes:
        rowptr = np.minimum(np.arange(n + 1, dtype=np.uint32), n - 1)
        col, gid = np.arange(1, n, dtype=np.uint32), C.c_uint64()
        assert lib.ga_server_add_graph(s, rowptr.ctypes.data_as(C.c_void_p), col.ctypes.data_as(C.c_void_p), n, n - 1,
                                       C.byref(gid)) == 0
        ids.append(gid)
    for i in requests:
        ticket, r = C.c_uint64(), RequestResult()
        assert lib.ga_server_submit(s, ids[i], 0, C.c_uint64(0), C.c_uint64(1), C.byref(ticket)) == 0
        assert lib.ga_server_wait(s, ticket, C.byref(r)) == 0 and r.status == 0
        results.append(r)
    stats = ServerStats()
    assert lib.ga_server_stats_get(s, C.byref(stats)) == 0 and lib.ga_server_destroy(s) == 0
    return results, stats


def test_recount_of_an_indexed_graph_reserves_nothing(lib):
    """A count on a resident graph whose index stands needs no more memory, whatever the estimate of an upload says: it
    evicts nothing."""
    a, b, much = 20011, 19001, 1 << 30
    used = serve_counts(lib, [a], [0, 0], much)[1].resident_bytes      # with the index
    upload = serve_counts(lib, [b], [0], much)[1].peak_reserved
    results, stats = serve_counts(lib, [a, b], [0, 0, 1, 1, 0, 0], used + upload)
    assert stats.evictions == 0 and [r.resident_hit for r in results] == [0, 1, 0, 1, 1, 1]
    assert stats.peak_reserved <= used + upload


def test_a_request_does_not_evict_its_own_graph(lib):
    """A second count, which needs the index that the first did without, makes room by evicting others, not the graph it is
    about to run on."""
    a, b, much = 30011, 29001, 1 << 30
    for n in (a, b):                                                   # both signatures known: first counts without index
        s, g = lib.graph(n=n)
        assert s == 0 and lib.ga_graph_prepare(g) == 0 and lib.ga_graph_destroy(g) == 0
    bare = serve_counts(lib, [a], [0], much)[1].resident_bytes
    upload = serve_counts(lib, [b], [0], much)[1].peak_reserved
    results, stats = serve_counts(lib, [a, b], [0, 1, 0], bare + upload)
    assert [r.resident_hit for r in results] == [0, 0, 1] and stats.evictions == 1
    assert stats.peak_reserved <= bare + upload


def test_autotuner_loads_what_it_times(lib):
    """The code of every kernel the autotuner times is loaded before the first timed launch."""
    s, g = lib.graph(n=777)
    assert s == 0
    lib.fake_reset()
    assert lib.ga_graph_prepare(g) == 0
    log = lib.log()
    loaded = {line.split()[1] for line in log if line.startswith("load")}
    timed = {line.split()[1] for line in log if line.startswith("launch") and "k_tc_" in line}
    assert len(timed) == 2 and timed == loaded
    assert lib.ga_graph_destroy(g) == 0


def test_every_captured_pass_has_its_own_queues(lib):
    s, g = lib.graph()
    assert s == 0 and lib.ga_graph_set_option(g, OPT_TC_KERNEL, C.c_int64(2)) == 0 and lib.ga_graph_prepare(g) == 0
    cleared = set()
    for _ in range(150):
        s, log = captured_call(lib, g, lambda g: CALLS["async"](lib, g))
        inside = [line for line in log if line.endswith("captured")]
        assert s == 0 and not [line for line in inside if line.startswith("alloc")]
        cleared |= {line for line in inside if line.startswith("memset") and str(C.addressof(TOTAL)) not in line}
    assert len(cleared) == 150
    assert lib.ga_graph_destroy(g) == 0 and lib.leaked() == 0
