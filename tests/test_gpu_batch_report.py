"""The launch shape that a batch reports is the one it runs: the FP64 tile
kernel has two threads a site (128 on a tile of 2 x 32) and three blocks an SM
whatever the number of events, the FP32 one 256 threads and one block. Saved
shapes that name one block an SM for it, as older files do, run the same."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

# argv: root, precision, number of events
_RUN = r'''
import sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import ipglasma_b200 as ipg
from test_gpu_step_kernels import make
prec, count = int(sys.argv[2]), int(sys.argv[3])
events = [make(prec, 32, 40 + k % 5) for k in range(count)]
with ipg.Batch(events) as b:
    r = b.tune()
    taken = []
    if r.from_cache:
        for blocks in (1, r.blocks_per_sm, r.blocks_per_sm + 1):
            try:
                b.set_shape(r.variant, blocks)
                taken.append(1)
            except ipg.IPGError:
                taken.append(0)
print("shape", r.from_cache, r.variant, r.tile_rows, r.threads_per_block, r.blocks_per_sm, r.grid,
      *taken)
'''


@pytest.mark.parametrize("prec,count,variant,rows,threads,blocks", [
    (0, 5, 2, 2, 128, 3), (0, 330, 2, 2, 128, 3), (1, 5, 3, 8, 256, 1)])
def test_report_of_the_tile_kernel(prec, count, variant, rows, threads, blocks, tmp_path):
    script, cache = tmp_path / "run.py", tmp_path / "shapes"
    script.write_text(_RUN)

    def run():
        out = subprocess.run([sys.executable, str(script), str(ROOT), str(prec), str(count)],
                             env={**os.environ, "IPG_TUNE_CACHE": str(cache)}, check=True,
                             capture_output=True, text=True, timeout=300).stdout
        return [int(x) for x in out.split("shape")[1].split()]

    assert run()[0] == 0  # timed, and saved for the next process
    (line,) = cache.read_text().splitlines()
    cache.write_text(f"{line.split()[0]} {variant} 1\n")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert run() == [1, variant, rows, threads, blocks, blocks * sms, 1, 1, 0]
