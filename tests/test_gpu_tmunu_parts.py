"""The parts of T^mu nu side by side (up to 128^2) and one after the other
(above) against the C restatement: one block, the last size of the first form
and the first of the second.

Bound: the links of the two sides differ by the Newton stop (1e-6) at most, and
a component is a sum of products of links of the order of the largest T^tautau;
the smallest components are above 1e-2 of it, so 1e-3 of a component's own
maximum holds with margin, and a part left out or finished twice is off by the
order of one."""
import numpy as np
import pytest

import ipglasma_b200 as ipg
from ipglasma_b200.synthetic import gaussian_blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ipg.FP64, ipg.FP32])
@pytest.mark.parametrize("N", [8, 128, 256])
def test_every_component_matches_the_restatement(N, prec, oracle_port):
    L, Ny = N * 0.078125, 2
    A, B = gaussian_blobs(N, L)
    cfg = ipg.Config(size=N, L=L, Ny=Ny, maxtime=0.1, precision=prec, seed=9)
    with ipg.Event(cfg) as ev:
        ev.set_g2mu(A, B)
        ev.use_device_noise()
        xi = [ev.draw_device_noise(k) for k in range(2)]
        ev.init_fields(allow_nonconverged=True)
        ev.run()
        T = ev.observables()[3]
    r = oracle_port.run_event(N, Ny, L, cfg.g, cfg.m, cfg.UVdamp, 0.1, A, B, xi[0], xi[1])
    for k in range(10):
        want = r["T10"][k]
        assert np.abs(T[k] - want).max() < 1e-3 * np.abs(want).max(), k
