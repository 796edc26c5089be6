"""Reading a field of an FP32 context widens the state on the context's stream
first; the read has to wait for that. Both reads see the same state, so they
are equal."""
import numpy as np
import pytest

import ipglasma_b200 as ipg
from ipglasma_b200.synthetic import gaussian_blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 32, 64])
def test_the_first_read_after_a_run_is_complete(N):
    L = N * 0.078125
    ev = ipg.Event(ipg.Config(size=N, L=L, Ny=2, maxtime=0.1, precision=ipg.FP32, seed=3))
    A, B = gaussian_blobs(N, L)
    ev.set_g2mu(A, B)
    ev.use_device_noise()
    for _ in range(8):
        ev.init_fields(allow_nonconverged=True)
        ev.run()
        first = ev.get_field(ipg.UX)
        assert np.array_equal(first, ev.get_field(ipg.UX))
    ev.close()
