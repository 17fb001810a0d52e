"""The pool of page-locked slots behind large copies (rg_stage.cpp), on the CPU: the file is
compiled against a CUDA runtime whose devices are host memory (fake_cudart.cpp), which counts the
sets of slots made and refuses what the real one refuses."""
import ctypes
import os
import signal
import subprocess
import threading
import time

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "raygen-renderer_b200", "csrc")
MB = 1 << 20


@pytest.fixture(scope="session")
def built(tmp_path_factory):
    if len(os.sched_getaffinity(0)) < 4:
        pytest.skip("copies are direct on few cores")
    out = tmp_path_factory.mktemp("stage") / "libstage.so"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + CSRC, "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "fake_cudart.cpp"), os.path.join(CSRC, "rg_stage.cpp"), "-o", str(out), "-Wl,-Bsymbolic",
                    "-lpthread"], check=True)
    lib = ctypes.CDLL(str(out))
    lib.fake_user.restype = ctypes.c_void_p
    lib.fake_user_end.argtypes = [ctypes.c_void_p]
    lib.fake_device.restype = ctypes.c_void_p
    lib.fake_round_trip.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t]
    lib.fake_upload.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_size_t]
    return lib


@pytest.fixture
def lib(built):
    user = built.fake_user()
    yield built
    built.fake_current(0)
    built.fake_capture_fails(0)
    built.fake_user_end(user)  # the last user: the pool is empty again


def data(mb, seed=0):
    return np.random.default_rng(seed).integers(0, 256, mb * MB, dtype=np.uint8)


def round_trip(lib, device, a):
    back = np.empty_like(a)
    assert lib.fake_round_trip(device, a.ctypes.data, back.ctypes.data, a.nbytes) == 0
    np.testing.assert_array_equal(a, back)


def test_copies_and_one_set(lib):
    """20 MB pays for a set; the copies after it use the same one."""
    before = lib.fake_sets_made()
    for k in range(5):
        round_trip(lib, 0, data(20, k)[k:])
    assert lib.fake_sets_made() - before == 1


def test_device_of_the_memory(lib):
    """A thread whose current device is another one than the handle's, as a program's reader
    threads are (their current device is 0 unless set): the copy is made all the same."""
    lib.fake_current(0)
    round_trip(lib, 1, data(20))
    round_trip(lib, 0, data(20))
    round_trip(lib, 1, data(20))


def test_sets_are_kept_per_device(lib):
    """Every device keeps the sets it made: a copy does not make one that is thrown away after it."""
    before = lib.fake_sets_made()
    for k in range(6):
        for device in range(4):
            lib.fake_current(device)
            round_trip(lib, device, data(20, k))
    assert lib.fake_sets_made() - before == 4


def test_concurrent_copies_make_no_more_sets_than_are_kept(lib):
    before = lib.fake_sets_made()
    a, errors = data(40), []

    def work():
        for _ in range(6):
            errors.append(lib.fake_upload(0, a.ctypes.data, a.nbytes))

    threads = [threading.Thread(target=work) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == [0] * 48
    assert lib.fake_sets_made() - before <= 2


def test_a_refused_capture_query_leaves_no_error_behind(lib):
    """Another thread's capture refuses the query of the default stream's state: the copy is a
    direct one, and the launch after it does not find the query's error."""
    lib.fake_capture_fails(1)
    round_trip(lib, 0, data(20))
    assert lib.fake_last_error() == 0


def test_one_core_copies_directly(lib):
    """A thread that may use one core or two makes no set: its copies would be slower for it."""
    cores = os.sched_getaffinity(0)
    before = lib.fake_sets_made()
    try:
        os.sched_setaffinity(0, {min(cores)})
        for k in range(3):
            round_trip(lib, 0, data(20, k))
    finally:
        os.sched_setaffinity(0, cores)
    assert lib.fake_sets_made() == before


def test_threads_are_kept_with_the_set(lib):
    """A copy starts no threads once its set is there, and they go with the set."""
    def threads():
        return len(os.listdir("/proc/self/task"))

    none = threads()
    round_trip(lib, 0, data(20))
    kept = threads()
    assert none < kept <= none + 7
    seen = []

    def watch():
        while not done.is_set():
            seen.append(threads())

    done = threading.Event()
    watcher = threading.Thread(target=watch)
    watcher.start()
    for k in range(10):
        round_trip(lib, 0, data(20, k))
    done.set()
    watcher.join()
    assert max(seen) <= kept + 1  # and the watcher
    second = lib.fake_user()
    lib.fake_user_end(second)
    assert threads() == kept


def test_threads_end_with_the_last_user(built):
    before = len(os.listdir("/proc/self/task"))
    user = built.fake_user()
    round_trip(built, 0, data(20))
    built.fake_user_end(user)
    assert len(os.listdir("/proc/self/task")) == before


@pytest.mark.filterwarnings("ignore:.*multi-threaded.*:DeprecationWarning")
def test_a_forked_child_may_end_its_users(built):
    """A child inherits the handles but no threads: closing the last one there returns."""
    user = built.fake_user()
    round_trip(built, 0, data(20))
    child = os.fork()
    if child == 0:
        built.fake_user_end(user)
        os._exit(0)
    for _ in range(200):
        pid, status = os.waitpid(child, os.WNOHANG)
        if pid:
            break
        time.sleep(0.05)
    else:
        os.kill(child, signal.SIGKILL)
        os.waitpid(child, 0)
        pytest.fail("the child hangs")
    assert status == 0
    round_trip(built, 0, data(20))
    built.fake_user_end(user)
