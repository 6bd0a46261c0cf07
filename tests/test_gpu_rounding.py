"""Float64 pushers against 80-bit arithmetic: the velocity after 1000 steps
through uniform fields (maps of equal node values), without half steps.  Every
rounding of a step at the size of the state adds an error of 2^-53 / sqrt(3) of it
(rms) at most; fields that turn the velocity make them independent, so that k of
them a step give sqrt(k / 3) 2^-53 sqrt(steps).  The bound is twice that with the
k of each update (``ROUNDINGS``): a term that is added to the state on its own,
where it could go with another, or a rounding that repeats from step to step,
shows as 2 to 10 times the error."""
import numpy as np
import pytest

from pypatools_b200 import Field
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker

pytestmark = pytest.mark.gpu
W = np.longdouble
C = W(299792458.0)
QM, SPEED, DT, STEPS = -1.75882001e11, 8.2e7, 5e-12, 1000      # 20 keV electrons
FIELDS = {"ExEyBz": ((2e5, -1e5, 0.0), (0.0, 0.0, 0.03)), "B": ((0.0, 0.0, 0.0), (0.01, -0.02, 0.03)),
          "full": ((2e5, -1e5, 3e4), (0.01, -0.02, 0.03)), "E": ((2e5, -1e5, 3e4), (0.0, 0.0, 0.0))}
# vay: u', the sum, 1 + t.t, its reciprocal, the product with it
# boris_rel: u-, the sum, u+ + kick, and t's 1/gamma
# vay_rel: gamma v + kick, the sum, the products with 1/gamma and with the clamp
ROUNDINGS = {"vay": 5, "boris_rel": 4, "vay_rel": 4}


def _dot(a, b):
    return np.sum(a * b, axis=-1, keepdims=True)


def _gamma_u(u):
    return np.sqrt(1 + _dot(u, u) / C ** 2)


def _vay(u, E, B, dt, qm):
    up = u + qm * dt * (E + np.cross(u / _gamma_u(u), B) / 2)
    tau = qm * dt / 2 * B
    tau2, us = _dot(tau, tau), _dot(up, tau) / C
    sigma = 1 + _dot(up, up) / C ** 2 - tau2
    t = tau / np.sqrt((sigma + np.sqrt(sigma ** 2 + 4 * (tau2 + us ** 2))) / 2)
    return (up + _dot(up, t) * t + np.cross(up, t)) / (1 + _dot(t, t))


def _boris_rel(u, E, B, dt, qm):
    um = u + qm * dt / 2 * E
    t = qm * dt / 2 / _gamma_u(um) * B
    return um + np.cross(um + np.cross(um, t), 2 * t / (1 + _dot(t, t))) + qm * dt / 2 * E


def _vay_rel(v, E, B, dt, qm):
    up = v / np.sqrt(1 - np.minimum(_dot(v, v) / C ** 2, W(0.9999))) + qm * dt * E
    tau = qm * dt / 2 * B
    tau2, q = _dot(tau, tau), _dot(up, tau) / C
    sigma = np.maximum(1 - _dot(up, up) / C ** 2, W(1e-10)) - tau2
    gn = np.sqrt((sigma + np.sqrt(sigma ** 2 + 4 * (tau2 + q * q))) / 2)
    t = tau / gn
    w = (up + np.cross(up + np.cross(up, t), 2 * t / (1 + _dot(t, t)))) / gn
    speed, top = np.sqrt(_dot(w, w)), W(0.9999) * C
    return np.where(speed >= top, w * top / speed, w)


def _uniform(v):
    g = np.array([-1e3, 0.0, 1e3])
    comps = {a: np.full((3, 3, 3), v[i]) for i, a in enumerate("xyz") if v[i] != 0.0}
    return Field.from_arrays({a: g for a in "xyz"}, comps) if comps else None


@pytest.mark.parametrize("alg,field", [("vay", "ExEyBz"), ("vay", "full"), ("boris_rel", "B"), ("vay_rel", "E")])
def test_error_is_that_of_its_roundings(cuda, alg, field):
    import torch
    dev = torch.device("cuda", 0)
    E, B = FIELDS[field]
    rng = np.random.default_rng(1)
    m = 256
    d = rng.normal(size=(m, 3))
    v = SPEED * d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.9, 1.0, (m, 1))
    tr = DeviceTracker(alg, QM, DeviceFields(_uniform(E), _uniform(B), "fp64", dev), m, STEPS, DT, STEPS, "fp64",
                       record=False, stagger=False, device=dev)
    r1, v1 = torch.zeros((m, 3), dtype=torch.float64, device=dev), torch.from_numpy(v).to(dev)
    tr.load(r1, v1)
    tr.advance(STEPS)
    tr.store(r1, v1)
    w, El, Bl = v.astype(W), np.array(E, dtype=W), np.array(B, dtype=W)
    u_state = alg != "vay_rel"
    if u_state:
        w = w / np.sqrt(1 - _dot(w, w) / C ** 2)
    step = {"vay": _vay, "boris_rel": _boris_rel, "vay_rel": _vay_rel}[alg]
    for _ in range(STEPS):
        w = step(w, El, Bl, W(DT), W(QM))
    if u_state:
        w = w / _gamma_u(w)
    err = np.linalg.norm((v1.cpu().numpy() - w).astype(float), axis=1) / np.linalg.norm(w.astype(float), axis=1)
    rms = np.sqrt(np.mean(err ** 2))
    assert rms <= 2 * np.sqrt(ROUNDINGS[alg] / 3) * 2.0 ** -53 * np.sqrt(STEPS), rms
