"""The staged leapfrog kernels at the edges of their tilings, to the bit
against kernels that share no staging code: the plain-load kernels
(IPG_FP32_KERNEL=pair, IPG_FP64_KERNEL=site) and, for a batch, each event on
its own. All run the same per-site arithmetic, so nothing may differ."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import ipglasma_b200 as ipg
from ipglasma_b200.synthetic import gaussian_blobs

pytestmark = pytest.mark.gpu
FIELDS = ("UX", "UY", "E1", "E2", "PHI", "PI")


def make(prec, N, seed):
    L = N * 0.078125
    ev = ipg.Event(ipg.Config(size=N, L=L, Ny=2, maxtime=0.1, precision=prec, seed=seed))
    A, B = gaussian_blobs(N, L)
    ev.set_g2mu(A, B)
    ev.use_device_noise()
    ev.init_fields(allow_nonconverged=True)
    return ev


_RUN = r'''
import sys, numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import ipglasma_b200 as ipg
from test_gpu_step_kernels import FIELDS, make
out = {}
for prec in (ipg.FP64, ipg.FP32):
    for N in (32, 64, 256):
        ev = make(prec, N, 3)
        ev.run()
        for f in FIELDS:
            out[f"{prec}{f}{N}"] = ev.get_field(getattr(ipg, f))
        ev.close()
np.savez(sys.argv[2], **out)
'''


def test_tiles_match_plain_loads(tmp_path):
    """One tile column (N = 32, every tile at two edges), two, and more tiles
    than an SM count."""
    root = str(Path(__file__).resolve().parent.parent)
    script = tmp_path / "run.py"
    script.write_text(_RUN)
    got = []
    for env in ({}, {"IPG_FP32_KERNEL": "pair", "IPG_FP64_KERNEL": "site"}):
        e = {k: v for k, v in os.environ.items() if not k.startswith("IPG_FP")}
        out = tmp_path / f"{len(got)}.npz"
        subprocess.run([sys.executable, str(script), root, str(out)], env={**e, **env},
                       check=True, timeout=600)
        got.append(np.load(out))
    assert len(got[0].files) == 36
    for k in got[0].files:
        assert np.array_equal(got[0][k], got[1][k]), k


@pytest.mark.parametrize("prec", [ipg.FP64, ipg.FP32])
@pytest.mark.parametrize("sizes", [(32,), (32, 64, 32), (64, 256, 32, 128), (32,) * 70])
def test_batch_matches_single_events(sizes, prec):
    """Fewer tiles than blocks, an event in the middle of a block's tiles, one
    that spans many blocks, and more descriptors than three blocks of an SM
    can hold beside their stages."""
    want = []
    for k, N in enumerate(sizes):
        ev = make(prec, N, 40 + k)
        ev.run()
        want.append([ev.get_field(getattr(ipg, f)) for f in FIELDS])
        ev.close()
    events = [make(prec, N, 40 + k) for k, N in enumerate(sizes)]
    with ipg.Batch(events) as b:
        b.run()
        for ev, w in zip(events, want):
            for f, x in zip(FIELDS, w):
                assert np.array_equal(ev.get_field(getattr(ipg, f)), x), (ev.N, f)
    for ev in events:
        ev.close()


@pytest.mark.parametrize("prec", [ipg.FP64, ipg.FP32])
def test_a_smaller_batch_beside_a_larger_one(prec):
    """The larger batch needs more shared memory a block; making the smaller
    one must not lower the limit of the kernel that both use."""
    large = [make(prec, 32, 40 + k) for k in range(12)]
    small = [make(prec, 32, 60)]
    with ipg.Batch(large) as b, ipg.Batch(small) as c:
        first = b.run()
        second = c.run()
    ev = make(prec, 32, 40)
    assert ev.run().E_T == first[0].E_T
    ev.close()
    assert np.isfinite(second[0].E_T)
    for ev in large + small:
        ev.close()
