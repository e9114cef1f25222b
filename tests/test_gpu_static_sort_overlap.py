"""wcsph_sort_keys_static keeps nothing between calls: calls may overlap on several
streams and be captured into a graph, also as the first call of a process."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import wcsph

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def keys_of(n, seed):
    k = np.random.default_rng(seed).integers(0, 1 << 40, n, dtype=np.int64)
    return torch.from_numpy(k).cuda(), np.argsort(k, kind="stable").astype(np.int32)


def test_overlapping_calls_on_streams():
    work = []
    for s in range(6):
        keys, want = keys_of(65536 - 777 * s, s)
        work.append((torch.cuda.Stream(), keys, torch.empty(len(want), dtype=torch.int32, device="cuda"), want))
    torch.cuda.synchronize()
    for _ in range(20):
        for st, keys, perm, _ in work:
            wcsph.sort_keys_static(keys.data_ptr(), len(keys), perm.data_ptr(), st.cuda_stream)
    torch.cuda.synchronize()
    for _, _, perm, want in work:
        assert np.array_equal(perm.cpu().numpy(), want)


CAPTURE = """
import sys
sys.path[:0] = sys.argv[1:]
import numpy as np, torch, wcsph
keys = torch.zeros(20000, dtype=torch.int64, device="cuda")
perm = torch.empty(20000, dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    wcsph.sort_keys_static(keys.data_ptr(), 20000, perm.data_ptr(), torch.cuda.current_stream().cuda_stream)
for seed in range(3):
    k = np.random.default_rng(seed).integers(0, 1 << 50, 20000, dtype=np.int64)
    keys.copy_(torch.from_numpy(k))
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(perm.cpu().numpy(), np.argsort(k, kind="stable"))
"""


def test_first_call_inside_a_capture():
    root = Path(__file__).resolve().parent.parent
    subprocess.run([sys.executable, "-c", CAPTURE, str(root / "fluid-simulation_b200")], check=True, timeout=300)
