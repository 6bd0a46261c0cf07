"""One step in one thread while another thread's rows wait for their track."""
import numpy as np
import pytest

from pypatools_b200 import Field, IonSpecies, PusherGPU
from pypatools_b200.pusher import HostStager

pytestmark = pytest.mark.gpu


def test_a_push_does_not_wait_for_queued_copies(cuda):
    torch = cuda
    g = np.linspace(-1.0, 1.0, 4)
    field = Field.from_arrays({a: g for a in "xyz"}, {"z": np.ones((4, 4, 4))})
    p = PusherGPU(IonSpecies("proton"), "boris")
    r, v = np.zeros((100, 3)), np.full((100, 3), 1e5)
    expect = p.push_batch(r, v, None, field, 1e-9)
    stager = HostStager.for_device(torch.device("cuda", 0))
    rows, host = torch.ones(1 << 20, dtype=torch.float64, device="cuda"), np.empty(1 << 20)
    other, ready = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(2_000_000_000)         # about a second
        ready.record(other)
    stager.copy(rows, host, ready)
    got = p.push_batch(r, v, None, field, 1e-9)
    waited = ready.query()
    stager.finish()
    assert not waited
    np.testing.assert_array_equal(got[0], expect[0])
    np.testing.assert_array_equal(got[1], expect[1])
    assert (host == 1.0).all()


def test_read_only_arrays_raise_no_warning(cuda):
    import warnings
    g = np.linspace(-1.0, 1.0, 4)
    field = Field.from_arrays({a: g for a in "xyz"}, {"z": np.ones((4, 4, 4))})
    r, v = np.zeros((3, 3)), np.full((3, 3), 1e5)
    r.flags.writeable = v.flags.writeable = False
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        r1, v1 = PusherGPU(IonSpecies("proton"), "boris").push_batch(r, v, None, field, 1e-9)
    assert np.isfinite(r1).all() and np.isfinite(v1).all()
