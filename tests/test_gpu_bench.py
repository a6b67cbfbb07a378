"""GPU: bench.py's step driven through patched blocks, where it asks each block how many launches a call takes."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


# launches per block: one for up to eight rows; above, three for the router, row preparation and matmul twice, combine
@pytest.mark.parametrize("config,tokens,per_block", [("c3", 2, 1), ("c1", 9, 8)])
def test_patched_blocks_and_plain_layers_report_the_same_launches(config, tokens, per_block):
    steps, layers = 3, 2
    for extra in ([], ["--via-patch"]):
        run = subprocess.run([sys.executable, "bench.py", "--config", config, "--tokens", str(tokens), "--layers", str(layers),
                              "--steps", str(steps), "--warmup", "3", "--repeats", "1", "--no-cpu-baseline", *extra],
                             cwd=ROOT, capture_output=True, text=True, timeout=300)
        assert run.returncode == 0, run.stderr[-2000:]
        line = json.loads(run.stdout.strip().splitlines()[-1])
        assert line["gpu_launches"] == steps * layers * per_block, extra
