"""Radius bounds whose min-plus tiles need about the 48 KB of shared memory that
a block has without asking for more, in a process that has not asked for more
yet (the limit stays raised once a larger radius has raised it)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

CODE = """
import hashlib, sys
import numpy as np, torch
from broxy_gb300 import _lib as L, api
mode, se, lanes, radii = int(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3]), [int(r) for r in sys.argv[4:]]
ctx, res = api.Context(0), 64
rng = np.random.default_rng(48)
X = torch.as_tensor(np.where(rng.random((res,) * 3) < 2e-4, 255, 0).astype(np.uint8).reshape(-1)).cuda()
d = api.make_desc(res)
for r in radii:
    out = torch.full_like(X, 0x5A)
    if lanes == 0:
        ctx.close(d, X, None, r, mode, se, out=out)
    else:
        ctx.batch_close_mesh([(d, X, None, r, out)], mode, se, 0, lanes, mesh=False)
    torch.cuda.synchronize()
    print(r, hashlib.sha1(out.cpu().numpy().tobytes()).hexdigest())
"""


def _run(mode, se, lanes, radii):
    r = subprocess.run([sys.executable, "-c", CODE, str(mode), str(se), str(lanes), *map(str, radii)], cwd=ROOT,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return dict(l.split() for l in r.stdout.splitlines())


@pytest.mark.parametrize("lanes", [0, -1])  # one closing; the grouped form of a batch
@pytest.mark.parametrize("mode,se", [(0, 0), (1, 0), (0, 1)])
def test_first_closing_near_the_limit(mode, se, lanes):
    radii = list(range(57, 67))
    assert _run(mode, se, lanes, radii) == {k: v for k, v in _run(mode, se, lanes, [90] + radii).items() if k != "90"}
