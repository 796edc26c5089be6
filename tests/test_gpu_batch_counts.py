"""FP64 batches of many small events. The tile kernel holds the descriptors of
87 events at a time, so its shape and what a batch may hold must not depend on
the number of events: a full window, one event more, windows that end in the
middle of a block's tiles, and more events than a block's shared memory could
describe at once. To the bit against the single-event kernel, which runs
the same per-site arithmetic."""
import numpy as np
import pytest

import ipglasma_b200 as ipg
from test_gpu_step_kernels import FIELDS, make

pytestmark = pytest.mark.gpu
TILES = 2  # the variant of the tile kernel in FP64
SEEDS = 5


@pytest.mark.parametrize("sizes", [(32,) * 87, (32,) * 88, (32, 64) * 70, (32,) * 330,
                                   (32,) * 1040], ids=lambda s: f"{len(s)}x{s[0]}-{s[-1]}")
def test_any_number_of_events_matches_single_events(sizes):
    want = {}
    for N in set(sizes):
        for k in range(SEEDS):
            ev = make(ipg.FP64, N, 40 + k)
            ev.run()
            want[N, k] = [ev.get_field(getattr(ipg, f)) for f in FIELDS]
            ev.close()
    events = [make(ipg.FP64, N, 40 + i % SEEDS) for i, N in enumerate(sizes)]
    with ipg.Batch(events) as b:
        b.set_shape(TILES, 1)
        b.run()
        for i, ev in enumerate(events):
            for f, x in zip(FIELDS, want[ev.N, i % SEEDS]):
                assert np.array_equal(ev.get_field(getattr(ipg, f)), x), (i, f)
    for ev in events:
        ev.close()
