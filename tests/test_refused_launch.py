"""Muon's Newton-Schulz iterations where their one launch is refused, since the process may use fewer SMs than the device has: as launches of their own, the
same bits.  The refusal is a fake of the runtime's call."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIM = Path(__file__).with_name("refused_launch.c")
PROGRAM = """
import sys
import numpy as np
from turbogpt_b200 import Config, ConfigEx, Native, bridge
depth, width = int(sys.argv[1]), int(sys.argv[2])
ex = ConfigEx.gpt(Config(depth=depth, context=64, batch=4, clip=1.0, ns_steps=5), width, width // 64, hidden_optimizer=bridge.HIDDEN_MUON)
with Native(ex) as engine:
    engine.set_weights((np.random.default_rng(1).standard_normal(engine.count) * .02).astype(np.float32))
    engine.set_data(np.random.default_rng(2).integers(0, 256, 1 << 14, dtype=np.uint8))
    for steps in (1, 3, 2):  # launched directly, captured, replayed
        engine.train(steps)
        losses = engine.training_losses(steps)
    np.save(sys.argv[3], np.concatenate([losses.ravel(), engine.weights()]))
"""


@pytest.mark.parametrize("depth,width", [(3, 192), (5, 960)])  # the families in one launch, and one by one
def test_refused_newton_schulz_launch(library, tmp_path, depth, width):
    shim = tmp_path / "refused.so"
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include", str(SHIM), "-o", str(shim), "-ldl"], check=True)
    results, refusals = [], []
    for preload in ("", str(shim)):
        out = tmp_path / f"{len(results)}.npy"
        done = subprocess.run([sys.executable, "-c", PROGRAM, str(depth), str(width), str(out)], cwd=SHIM.parents[1], capture_output=True, text=True,
                              timeout=300, env={**os.environ, "LD_PRELOAD": preload, "PYTHONPATH": str(SHIM.parents[1])})
        assert done.returncode == 0, done.stderr
        results.append(np.load(out))
        refusals.append(done.stderr.count("refused\n"))
    assert refusals == [0, 1]  # asked for once
    np.testing.assert_array_equal(*results)
