"""The host code where a CUDA call fails, and where it has to count or to wait.

The library's own objects are linked with tests/fake_cuda.cpp, a runtime whose
kernels do nothing and whose calls fail when a test says so: no GPU is used and
none is needed.  A test runs in a process of its own, so that a crash or a hang
of the library is a failed test.
"""
import glob
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT

PRELUDE = """
import ctypes, os, sys, time
import numpy as np
sys.path.insert(0, {root!r})
import ap26_b200 as A
A.LIB_PATH = {lib!r}
A.lib = fake = A._load()
fake.fake_fail.argtypes = [ctypes.c_char_p] + [ctypes.c_int] * 3
fake.fake_read_back.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_ulonglong]
OOM, OTHER = 2, 999        # cudaErrorMemoryAllocation, cudaErrorUnknown
ALL = 1 << 30
def fail(call, skip=0, times=ALL, code=OTHER):
    fake.fake_fail(call.encode(), skip, times, code)
"""


def _built_objects():
    """The library's objects, brought up to date as the build does it."""
    spec = importlib.util.spec_from_file_location(
        "ap26_build", os.path.join(ROOT, "ap26_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    objs = [os.path.join(build.BUILD, f) for f in ("ap26_capi.o", "ap26_host.o")]
    srcs = glob.glob(os.path.join(build.CSRC, "*")) + [os.path.join(ROOT, "include", "ap26.h")]
    if not all(build._newer(o, srcs) for o in objs):
        if not os.path.exists(build.NVCC):
            pytest.skip("the library's objects are not built")
        build.build()
    return objs


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no host C++ compiler or no CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "libap26_fake.so")
    subprocess.run(["g++", "-O1", "-fPIC", "-shared", "-std=c++17", "-Wl,-Bsymbolic", "-I", inc,
                    os.path.join(ROOT, "tests", "fake_cuda.cpp")] + _built_objects() +
                   ["-lpthread", "-o", so], check=True)
    return so


@pytest.fixture
def child(fake_lib):
    def run(code, timeout=60):
        p = subprocess.run([sys.executable, "-c",
                            PRELUDE.format(root=ROOT, lib=fake_lib) + textwrap.dedent(code)],
                           capture_output=True, text=True, timeout=timeout)
        assert p.returncode == 0, (p.returncode, p.stdout, p.stderr)
        return p.stdout
    return run


def test_chain_walks_after_the_job_set_could_not_grow(child):
    """A batch of more K than the job set holds frees it to make a larger one.
    Where that fails the batch fails, and the calls after it get a set of their
    own or an error: chain_batch keeps its error flags there."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        n = np.arange(1, 2001, 2, dtype=np.int64)
        ctx.chain_batch(1, n)
        fail("cudaMalloc", code=OOM)
        try:
            ctx.sieve_count(range(1, 200), 0)
            raise SystemExit("no memory, and a count all the same")
        except A.AP26Error as e:
            assert e.code == A.E_CUDA
        for _ in range(2):
            try:
                ctx.chain_batch(1, n)
                raise SystemExit("no memory, and a walk all the same")
            except A.AP26Error as e:
                assert e.code == A.E_CUDA
        fail("cudaMalloc", times=0)
        try:
            ctx.chain_batch(1, n)
        except A.AP26Error:               # the failed call's own pending error
            pass
        ctx.chain_batch(1, n)
        ctx.close()
    """)


def test_noalloc_takes_the_errors_of_its_own_launches(child):
    """A pending error is the caller's: the call that finds one launches nothing.
    So a call that fails leaves none of its own, whichever launch failed, and
    launches nothing after it."""
    child("""
        Ks = (ctypes.c_int32 * 2)(1, 2)
        out = (ctypes.c_int64 * 2)()
        def count():
            before = fake.fake_launches()
            rc = A.lib.ap26_sieve_count_noalloc(0, Ks, 2, 0, out, None)
            return rc, fake.fake_launches() - before
        rc, launches = count()
        assert rc == A.OK and launches == 2 + 2 * 7 + 1
        for call, steps in (("cudaMemsetAsync", 2), ("cudaLaunchKernel", launches)):
            for i in range(steps):
                fail(call, skip=i, times=1)
                rc, done = count()
                assert rc == A.E_CUDA, (call, i)
                assert done == (i if call == "cudaLaunchKernel" else 2 + 7 * i), (call, i, done)
                assert fake.cudaPeekAtLastError() == 0, (call, i)
                assert count() == (A.OK, launches), (call, i)
    """)


def test_launches_of_long_calls_are_counted(child):
    """stats.launches of a call that is cut in slices counts each slice's kernel;
    a range's candidates behind the first 2^20 take a kernel for each 2^20."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        def launched(call):
            before = fake.fake_launches()
            st = call()
            return fake.fake_launches() - before, st.launches
        for n, slices in ((1, 1), (1 << 17, 1), (1 << 20, 1), ((1 << 20) + 1, 2), (5 << 20, 5)):
            N = np.full(n, 9, np.uint64)
            assert launched(lambda: ctx.sprp_batch(N)[1]) == (slices, slices), n
        n = 3_000_001
        a = np.full(n, 2, np.uint32)
        assert launched(lambda: ctx.sprp_bases(np.full(n, 9, np.uint64), a)[1]) == (5, 5)
        assert launched(lambda: ctx.chain_batch(1, np.full(n, 9, np.int64))[2]) == (5, 5)
        reps, fin, st = np.zeros(n, A._AP), np.zeros(n, "V56"), A.Stats()
        def report():
            A.lib.ap26_report_batch(ctx.h, A._ptr(reps), n, A._ptr(fin), None, ctypes.byref(st))
            return st
        assert launched(report) == (21, 21)
        DEVSTATE, CAND_COUNT = 128, 40
        for n, more in ((0, 0), (1 << 20, 0), ((1 << 20) + 1, 1), (5 << 20, 4)):
            with A.Context(0, cand_ring_log2=23) as big:
                fake.fake_read_back(DEVSTATE, CAND_COUNT, n)
                call = lambda: big.sieve_range(1, 0, 0, A.N53_PER_K, cap=1 << 23)
                assert launched(lambda: call()[1]) == (2 + more, 2 + more), n
        ctx.close()
    """)


def test_threads_of_a_long_call_do_not_spin_while_one_is_late(child):
    """A slice's kernel starts when every thread has copied its part.  A thread
    that the system holds back keeps the others waiting: they wait asleep, and
    leave it their share of the processor time."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        N = np.full(1 << 22, 9, np.uint64)
        ctx.sprp_batch(N)                       # starts the threads
        fake.fake_slow_copy(1000)
        cpu, wall = time.process_time(), time.perf_counter()
        ctx.sprp_batch(N)
        cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
        assert wall >= 1, wall
        assert cpu < 0.5 * wall, (cpu, wall)
        ctx.close()
    """)


def test_one_thread_of_a_long_call_waits_for_the_device(child):
    """A long call may wait for work that is queued before it, such as a serving
    slice.  The runtime's wait spins: one thread takes it, the others sleep."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        N = np.full(1 << 22, 9, np.uint64)
        ctx.sprp_batch(N)                       # starts the threads
        fake.fake_busy_device(200)
        cpu, wall = time.process_time(), time.perf_counter()
        ctx.sprp_batch(N)                       # four slices
        cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
        assert wall >= 0.8, wall
        assert cpu < 1.5 * wall, (cpu, wall)
        ctx.close()
    """)


def test_threads_of_a_long_call_wake_in_time(child):
    """A slice's results are copied out as soon as they are there, also where its
    kernel takes some milliseconds, as that of 140000 reports does: no thread
    sleeps for a time, each waits until it is woken."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        N = np.full(1 << 20, 9, np.uint64)      # one slice
        ctx.sprp_batch(N)
        for ms in (2, 6, 20):
            fake.fake_busy_device(ms)
            before = fake.fake_sleeps()
            ctx.sprp_batch(N)
            assert fake.fake_sleeps() == before, ms
        ctx.close()
    """)


def test_long_calls_with_memory_for_one_set_of_buffers(child):
    """The context has one set of buffers from the start.  A long call uses three;
    where there is no memory for the others it goes through those there are, and
    a later one gets the rest."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        n = (5 << 20) + 3
        N = np.arange(n, dtype=np.uint64)
        a = np.full(n, 2, np.uint32)
        for call in ("cudaMalloc", "cudaHostAlloc"):
            for skip in (0, 1):                  # the first or the second buffer
                fail(call, skip=skip, code=OOM)
                assert ctx.sprp_batch(N)[1].launches == 6
                assert ctx.sprp_bases(N, a)[1].launches == 8
                fail(call, times=0)
        assert ctx.sprp_batch(N)[1].launches == 6
        ctx.close()
    """)


def test_long_calls_need_no_host_memory_of_their_own(child):
    """No exception leaves a C entry point: a long call allocates nothing on the
    host but its threads, and does without those."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        N = np.arange(5 << 20, dtype=np.uint64)
        v, st = np.empty(len(N), np.uint8), A.Stats()
        fake.fake_no_host_memory(1)
        rc = A.lib.ap26_sprp_batch(ctx.h, A._ptr(N), len(N), A._ptr(v), ctypes.byref(st))
        fake.fake_no_host_memory(0)
        assert rc == A.OK and st.launches == 5
        ctx.close()
    """)


def test_a_forked_child_lets_go_of_the_context(child):
    """The host threads of long calls are not there in a forked child: a context
    that goes there, as an interpreter's last act, waits for none of them."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        ctx.sprp_batch(np.full(1 << 22, 9, np.uint64))
        pid = os.fork()
        if pid == 0:
            ctx.close()
            os._exit(0)
        end = time.time() + 20
        while time.time() < end:
            done, status = os.waitpid(pid, os.WNOHANG)
            if done:
                break
            time.sleep(0.01)
        else:
            os.kill(pid, 9)
            os.waitpid(pid, 0)
            raise SystemExit("the child hangs")
        assert status == 0, status
        ctx.sprp_batch(np.full(1 << 22, 9, np.uint64))
        ctx.close()
    """)


def test_reports_with_numbers_beyond_their_fields_reach_the_library(child):
    """k, K, first and n go to the library as C integers of their fields, whatever
    was given: a status for each report, and no exception of the binding's."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        seen = []
        real = fake.ap26_report_batch
        class Lib:
            def __getattr__(self, name):
                return getattr(fake, name)
            def ap26_report_batch(self, h, aps, n, *rest):
                buf = aps if isinstance(aps, ctypes.Array) else ctypes.cast(aps, ctypes.POINTER(A.AP))
                seen.append([(buf[i].k, buf[i].K, buf[i].first, buf[i].n) for i in range(n)])
                return real(h, aps, n, *rest)
        A.lib = Lib()
        rows = [(10, 1 << 31, 31, 7), (1 << 32, 5, 1 << 63, -1), (-1, -(1 << 31) - 1, -(1 << 63), 2),
                (10.0, 3, np.int64(37)), (11, 4, (1 << 64) + 3, 1 << 64)]
        rc, fin, h = ctx.report_batch(rows, result_hash=5)
        assert len(fin) == 5
        want = [A.AP(int(r[0]), int(r[1]), int(r[2]), int(r[3]) if len(r) > 3 else 0) for r in rows]
        assert seen == [[(w.k, w.K, w.first, w.n) for w in want]]
        assert ctx.report_batch([])[1] == []
        ordinary = [(10 + i, 366384, 10**15 + i, 10**15) for i in range(40)]
        ctx.report_batch(ordinary)
        assert seen[-1] == ordinary
        ctx.close()
    """)


@pytest.mark.parametrize("K", [43241061, 61 * 67 * 71 * 73, 149 * 151 * 157 * 113, 199 * 541,
                               523 * 541, 139 * 149 * 151])
def test_a_range_is_sieved_once_whatever_divides_k(child, K):
    """The binding makes room for the candidates it expects and sieves again where
    they are more: every sieve prime that divides K counts, so they are not."""
    child(f"""
        K, starts = {K}, 2_000_000
        rooms = []
        class Lib:
            def __getattr__(self, name):
                return getattr(fake, name)
            def ap26_sieve_range(self, h, K, shift, q0, q1, cand, cap, n, st):
                rooms.append(cap)
                n._obj.value = found
                return A.OK if found <= cap else A.E_CAPACITY
        density = 36.9e6 / A.N53_PER_K           # of a K that no sieve prime divides
        for p in range(61, 542):
            if K % p == 0 and all(p % d for d in range(2, 24)):
                density *= (p - 1) / (p - 24)
        found = int(1.1 * density * starts)
        ctx = A.Context(0, cand_ring_log2=12)
        A.lib = Lib()
        cand, st = ctx.sieve_range(K, 0, 0, starts)
        assert len(cand) == found and len(rooms) == 1, (rooms, found)
        ctx.close()
    """)


def test_the_version_tells_the_scratch_size_and_late_items(child):
    """A program asks ap26_version() which of the header's figures hold: the size
    of the allocation-free scratch, and what late_items counts for a whole K."""
    with open(os.path.join(ROOT, "include", "ap26.h")) as f:
        size = int(re.search(r"#define AP26_NOALLOC_SCRATCH_BYTES (\d+)", f.read()).group(1))
    out = child("print(A.lib.ap26_version())")
    assert {10100: 2349440, 10200: 15591200}[int(out)] == size


def test_a_long_call_that_fails_leaves_the_next_one_alone(child):
    """Whichever step of whichever thread fails: the call ends with AP26_E_CUDA, no
    thread hangs, and none keeps the error for a later call to find."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        N = np.full(5 << 20, 9, np.uint64)      # five slices, eight threads
        calls = 0
        for call in ("cudaMemcpyAsync", "cudaEventRecord", "cudaStreamWaitEvent",
                     "cudaEventSynchronize", "cudaLaunchKernel", "cudaSetDevice"):
            for skip in (0, 1, 3, 4, 7, 12, 20, 33):
                fail(call, skip=skip, times=1)
                try:
                    ctx.sprp_batch(N)
                except A.AP26Error as e:
                    assert e.code == A.E_CUDA, (call, skip)
                    calls += 1
                fail(call, times=0)
                for _ in range(4):
                    assert ctx.sprp_batch(N)[1].launches == 5
        assert calls > 24, calls
        ctx.close()
    """, timeout=120)


def test_rings_that_could_not_be_resized_are_made_again_before_use(child):
    """set_opts frees the candidate rings to make others.  Where that fails, no
    kernel gets the pointers that are left: the next call makes the rings again,
    of the size the options still have, or fails."""
    child("""
        ctx = A.Context(0, cand_ring_log2=13)
        uses = [lambda: ctx.sieve_range(1, 0, 0, 1000), lambda: ctx.search_k(43241061),
                lambda: ctx.search_batch([(1, 43241061, 43241062, 0)])]
        for use in uses:
            for skip in (0, 1):                  # the first or the second ring
                fail("cudaMalloc", skip=skip, code=OOM)
                try:
                    ctx.set_opts(cand_ring_log2=14)
                    raise SystemExit("no memory, and rings all the same")
                except A.AP26Error as e:
                    assert e.code == A.E_CUDA
                assert ctx.opts["cand_ring_log2"] == 13
                before = fake.fake_launches()
                try:
                    use()
                    raise SystemExit("no rings, and a run all the same")
                except A.AP26Error as e:
                    assert e.code == A.E_CUDA
                assert fake.fake_launches() == before
                fail("cudaMalloc", times=0)
                use()
                assert fake.fake_launches() > before
        assert ctx.set_opts(cand_ring_log2=14)["cand_ring_log2"] == 14
        ctx.close()
    """)


def test_serving_buffers_that_could_not_be_made_are_made_later(child):
    """The first admission makes serving's buffers.  Where one of them fails the
    admission fails, and a later one makes what is missing: no slice runs without."""
    child("""
        for call in ("cudaMalloc", "cudaHostAlloc"):
            for skip in range(24):
                ctx = A.Context(0, cand_ring_log2=12)
                fail(call, skip=skip, code=OOM)
                made = ctx.serve_submit(1, 43241061, 43241063, 0)
                assert made in (A.OK, A.E_CUDA), (call, skip)
                fail(call, times=0)
                if made != A.OK:
                    assert ctx.serve_submit(1, 43241061, 43241063, 0) == A.OK
                for _ in range(4):
                    ctx.serve_step()
                ctx.close()
                if made == A.OK:
                    break
            assert made == A.OK and skip > 3, (call, skip)
    """)


def test_serving_goes_on_once_there_is_memory_for_its_rings(child):
    """A step that finds no memory for the candidate rings fails and takes no K: the
    unit's K are all searched once there is some."""
    child("""
        ctx = A.Context(0, cand_ring_log2=12)
        assert ctx.serve_submit(1, 43241061, 43241063, 0) == A.OK
        fail("cudaMalloc", code=OOM)
        try:
            ctx.set_opts(cand_ring_log2=13)
            raise SystemExit("no memory, and rings all the same")
        except A.AP26Error:
            pass
        for _ in range(3):
            try:
                ctx.serve_step()
                raise SystemExit("no rings, and a step all the same")
            except A.AP26Error as e:
                assert e.code == A.E_CUDA
        fail("cudaMalloc", times=0)
        ctx.serve_step()
        assert ctx.serve_step() == 0             # no unit left: all of its K are done
        ctx.close()
    """)
