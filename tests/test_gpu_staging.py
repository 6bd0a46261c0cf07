"""Staged copies of ordinary numpy arrays (``ppt_stager_*``): every byte
arrives, for sizes around a piece, a slot and the whole ring, in both
directions, while other work is queued, and from several threads at once."""
import threading

import numpy as np
import pytest

from pypatools_b200 import _lib

pytestmark = pytest.mark.gpu
KIB = 1 << 10
# below, at and above one handed-over piece; slots of 1 MiB, rings of 8; ragged ends
SIZES = [1, 8, 255 * KIB, 256 * KIB, 256 * KIB + 1, 1 << 20, (1 << 20) + 4097, (8 << 20) - 1, 8 << 20, (37 << 20) + 13]


def _stager(torch, **kw):
    from pypatools_b200.pusher import HostStager
    return HostStager(torch.device("cuda", 0), chunk=1 << 20, slots=8, threads=3, **kw)


@pytest.mark.parametrize("nbytes", SIZES)
def test_round_trip(cuda, nbytes):
    torch = cuda
    st = _stager(torch)
    src = np.random.default_rng(nbytes).integers(0, 256, nbytes, dtype=np.uint8)
    dev = torch.full((nbytes,), 7, dtype=torch.uint8, device="cuda")
    st.upload(src, dev)
    expect = src.copy()
    src[:] = 0                                  # read when upload returned
    dev += 1                                    # queued after the copy, on the current stream
    dst = np.full(nbytes, 255, dtype=np.uint8)
    ev = torch.cuda.Event()
    ev.record()
    st.copy(dev, dst, ev)
    st.finish()
    np.testing.assert_array_equal(dst, expect + np.uint8(1))
    with pytest.raises(ValueError):
        st.upload(src, dev[1:] if nbytes > 1 else torch.empty(2, dtype=torch.uint8, device="cuda"))
    _lib.check(_lib.load().ppt_stager_destroy(st.handle))


def test_several_threads_share_a_ring(cuda):
    torch = cuda
    st = _stager(torch)
    out = {}

    def work(k):
        stream = torch.cuda.Stream()
        rng = np.random.default_rng(k)
        ok = True
        for i in range(6):
            a = rng.normal(size=(k + 1) * 70_001)
            with torch.cuda.stream(stream):
                d = torch.empty(a.shape, dtype=torch.float64, device="cuda")
                st.upload(a, d, stream)
                d *= 2.0
                ev = torch.cuda.Event()
                ev.record(stream)
            b = np.empty_like(a)
            st.copy(d, b, ev)
            st.finish()
            ok = ok and np.array_equal(b, 2.0 * a)
        out[k] = ok

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert out == {k: True for k in range(4)}


def test_arguments():
    lib = _lib.load()
    out = _lib.c_void_p()
    for slot, n, threads in ((100, 4, 1), (4096, 1, 1), (4096, 4, 0)):
        assert lib.ppt_stager_create(slot, n, threads, None, out) == -1
    assert lib.ppt_stager_finish(None) == -1 and lib.ppt_stager_destroy(None) == 0
    assert lib.ppt_stager_upload(None, None, None, 8, None) == -1
