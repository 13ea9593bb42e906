"""One switch selects the kernels of the embedding gradient, whoever asks: set from the environment when the functions are imported,
by `set_deterministic_embedding_grad` after that, before or after the extension is loaded."""
import os
import subprocess
import sys

import pytest

SET, CLEAR = "os.environ['SSB_EMBEDDING_GRAD_ATOMICS'] = '1'", "os.environ.pop('SSB_EMBEDDING_GRAD_ATOMICS')"
IMPORT, LOAD = "from superscaler_b200.ops import functional as F, native", "native.ext()"


@pytest.mark.parametrize("steps,in_order", [
    ([IMPORT, LOAD], True), ([SET, IMPORT, LOAD], False),
    ([IMPORT, SET, LOAD], True), ([SET, IMPORT, CLEAR, LOAD], False),        # the environment changes in between
    ([IMPORT, "F.set_deterministic_embedding_grad(False)", LOAD], False),
    ([SET, IMPORT, "F.set_deterministic_embedding_grad(True)", LOAD], True),
    ([IMPORT, LOAD, "F.set_deterministic_embedding_grad(False)"], False),
])
def test_the_switch_is_the_extensions(steps, in_order):
    env = {k: v for k, v in os.environ.items() if k != "SSB_EMBEDDING_GRAD_ATOMICS"}
    code = "\n".join(["import os", *steps, "print(native.ext().embedding_in_order())"])
    run = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    if "native extension unavailable" in run.stderr:
        pytest.skip("extension not built")
    assert run.stdout.split()[-1:] == [str(in_order)], run.stderr
