"""The mixed form's FP32 engines give the bits of the engines that they replaced:
its error estimate on large grids and the largest constraint of small ones are
rounding noise, and step sequences follow them.  The recorded checksums hold for the
compiler that made them too: a failure after a change of compiler alone says that
it contracts products another way."""
import json
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, str(Path(__file__).parent / "golden"))
import make_mixed_bits as M  # noqa: E402


@pytest.mark.parametrize("n", M.GRIDS, ids=M.key)
def test_bits(n):
    from instaheat_gb300 import gpu
    assert M.checksums(gpu, n) == json.loads(M.FILE.read_text())[M.key(n)]
