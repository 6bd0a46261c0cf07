"""The staging of host copies without a GPU: csrc/staging.cu against a stand-in
for the CUDA runtime (tests/stager_host), and the Python side's references."""
import shutil
import subprocess
import weakref
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
REPO = HERE.parent


def _compile(folder, *flags):
    """The cases' program.  staging.cu is copied beside the stand-in, so that
    its quoted include finds that first."""
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    for name in ("ppt_internal.cuh", "main.cpp"):
        shutil.copy(HERE / "stager_host" / name, folder / name)
    shutil.copy(REPO / "pypatools_b200" / "csrc" / "staging.cu", folder / "staging.cu")
    exe = folder / "cases"
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", *flags, "-I", str(REPO / "include"), str(folder / "main.cpp"),
                    "-o", str(exe), "-lpthread"], check=True, capture_output=True, text=True)
    return exe


@pytest.fixture(scope="module")
def cases(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("stager"))


@pytest.mark.parametrize("case", ["refused_download", "refused_upload", "error_of_its_caller", "destroyed_twice",
                                  "several_callers"])
def test_stager(cases, case):
    res = subprocess.run([str(cases), case], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stderr


class _FakeLib:
    def __init__(self):
        self.finished = 0

    def ppt_stager_download(self, *a):
        return 0

    def ppt_stager_finish(self, handle):
        self.finished += 1
        return 0


def _stager():
    import threading
    from pypatools_b200.pusher import HostStager
    st = object.__new__(HostStager)
    st.lib, st.handle, st._copies, st._copies_lock = _FakeLib(), 1, [], threading.Lock()
    return st


def test_a_copy_keeps_both_ends_until_finish():
    import torch
    st = _stager()
    src, dst = torch.zeros(10, dtype=torch.float64), np.empty(10)
    ends = weakref.ref(src), weakref.ref(dst)
    st.copy(src, dst)
    del src, dst
    assert all(r() is not None for r in ends)
    st.finish()
    assert all(r() is None for r in ends)


def test_an_interrupted_track_waits_for_its_rows(monkeypatch):
    """A track that ends with an exception after rows were queued."""
    import contextlib
    import torch
    from pypatools_b200 import IonSpecies, pusher
    st = _stager()

    class Tracker:
        active = None

        def __init__(self, alg, qm, df, m, nsteps, dt, rec, *a, **k):
            self.r_hist = torch.zeros((nsteps // rec + 1, m, 3), dtype=torch.float64)
            self.v_hist = self.r_hist.clone()

        def load(self, r, v):
            pass

        def run(self, nsteps, chunk, sort_every=0, after_launch=None):
            after_launch(nsteps // 2)
            raise KeyboardInterrupt

    class Fields:
        device = torch.device("cpu")

    class Event:
        cuda_event = 0

        def record(self, stream):
            pass

    monkeypatch.setattr(pusher, "DeviceTracker", Tracker)
    monkeypatch.setattr(pusher, "_torch", lambda: torch)
    monkeypatch.setattr(pusher.HostStager, "for_device", classmethod(lambda cls, device: st))
    monkeypatch.setattr(pusher.PusherGPU, "_device_fields", lambda self, e, b: Fields)
    monkeypatch.setattr(pusher.PusherGPU, "_upload", staticmethod(lambda a, device: torch.from_numpy(a)))
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: None)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    p = pusher.PusherGPU(IonSpecies("proton"), "boris")
    with pytest.raises(KeyboardInterrupt):
        p.track_batch(np.zeros((5, 3)), np.ones((5, 3)), None, None, 10, 1e-10)
    assert st.lib.finished == 1 and not st._copies


def test_no_data_race(tmp_path):
    probe = tmp_path / "probe"
    (tmp_path / "probe.cpp").write_text("int main() { return 0; }\n")
    built = shutil.which("g++") and subprocess.run(["g++", "-fsanitize=thread", str(tmp_path / "probe.cpp"), "-o",
                                                    str(probe)], capture_output=True).returncode == 0
    if not built or subprocess.run([str(probe)], capture_output=True).returncode != 0:
        pytest.skip("no ThreadSanitizer here")
    exe = _compile(tmp_path, "-fsanitize=thread")
    for _ in range(3):
        res = subprocess.run([str(exe), "several_callers"], capture_output=True, text=True, timeout=300)
        if "unexpected memory mapping" in res.stderr:          # the system's address layout, at random
            pytest.skip("no ThreadSanitizer here")
        assert res.returncode == 0, res.stderr[:4000]


def test_a_device_has_one_stager(monkeypatch):
    import threading
    import time
    from pypatools_b200.pusher import HostStager
    made = []

    def init(self, device):
        made.append(self)
        time.sleep(0.05)

    monkeypatch.setattr(HostStager, "__init__", init)
    monkeypatch.setattr(HostStager, "_by_device", {})
    threads = [threading.Thread(target=HostStager.for_device, args=("cuda:0",)) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1


def test_a_dropped_stager_is_destroyed(monkeypatch):
    import contextlib
    import torch
    from pypatools_b200 import pusher

    class Lib(_FakeLib):
        destroyed = []

        def ppt_stager_create(self, chunk, slots, threads, stream, out):
            out.value = 77
            return 0

        def ppt_stager_destroy(self, handle):
            self.destroyed.append(handle)
            return 0

    class Stream:
        cuda_stream = 5

        def __init__(self, device):
            pass

    lib = Lib()
    monkeypatch.setattr(pusher._lib, "load", lambda: lib)
    monkeypatch.setattr(pusher, "_torch", lambda: torch)
    monkeypatch.setattr(torch.cuda, "Stream", Stream)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    st = pusher.HostStager(torch.device("cuda", 0))
    assert st.handle == 77 and not lib.destroyed
    del st
    assert lib.destroyed == [77]
