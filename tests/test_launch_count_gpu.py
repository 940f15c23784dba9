"""bem200_launch_count counts every kernel once: an inverse reports as many
launches when its kernels are issued directly as when its graph is replayed."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import torch
from mnpbem_b200 import _native as nat
L = nat.lib()
for code, dt in ((nat.C64, torch.complex64), (nat.C128, torch.complex128)):
    for n in (40, 64, 200, 300, 900):
        A = torch.randn((n, n), dtype=dt, device="cuda") / n ** 0.5 + 4 * torch.eye(n, dtype=dt, device="cuda")
        scr = torch.empty(int(L.bem200_inverse_nopiv_workspace_size(code, n)), dtype=torch.uint8, device="cuda")
        ws, info = torch.empty(1, dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        before = int(L.bem200_launch_count())
        nat.call("bem200_inverse_nopiv", code, 0, n, nat.ptr(A), n, nat.ptr(ws), 0, nat.ptr(scr), 1e-2, nat.ptr(info),
                 nat.stream_ptr())
        print(n, int(L.bem200_launch_count()) - before)
torch.cuda.synchronize()
"""


def _counts(no_graphs):
    env = dict(os.environ, BEM200_NO_GRAPHS="1" if no_graphs else "0")
    return subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env=env, capture_output=True, text=True, check=True,
                          timeout=300).stdout


def test_direct_and_replayed_launches_count_alike(cuda):
    direct, replayed = _counts(True), _counts(False)
    assert len(direct.split("\n")) > 10 and direct == replayed, (direct, replayed)
