"""A call of so many substeps that the escapes are no longer counted in the substeps'
barrier word: the same trajectory as two calls of half as many, which count them."""
import numpy as np
import pytest

from helpers import SCENARIOS, gpu_frame_step, initial_state, to_gpu_state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_one_long_call_equals_two(golden32):
    g = golden32
    fs = gpu_frame_step(g, "small", torch.float32)
    k, dt = SCENARIOS["small"][2], SCENARIOS["small"][3]
    grid = fs.info()["grid_blocks"]
    half = int(1.6e7 / (k * grid)) + 1  # two halves are above the 3e7 substeps x CTAs of a counted call, one is below
    K = 2 * half
    assert K * k * grid >= 3e7 > half * k * grid
    st0, sh0 = to_gpu_state(*initial_state(g, "small", np.float32), torch.float32)
    # over the ice and back, again and again, so that elements keep leaving their margins
    eta = sh0.eta.cpu().numpy().astype(np.float64)
    t = np.arange(K + 1) * dt
    track = np.tile(eta, (K + 1, 1))
    track[:, :2] += (30.0 - 30.0 * np.cos(t / 15.0))[:, None] * np.array([np.cos(eta[2]), np.sin(eta[2])])
    rows = torch.as_tensor(np.concatenate([track[:-1], track[1:]], 1), dtype=torch.float32, device="cuda")
    vw = torch.zeros((K, st0.positions.shape[0], 2), dtype=torch.float32, device="cuda")
    whole, ship, _ = fs.scan_segment(st0, sh0, rows, vw, history=False)
    escaped = fs.info()["escaped_total"]
    a, b, _ = fs.scan_segment(st0, sh0, rows[:half].contiguous(), vw[:half], history=False)
    a, b, _ = fs.scan_segment(a, b, rows[half:].contiguous(), vw[half:], history=False)
    fs.close()
    assert whole.elem_active.any() and escaped > 100
    for x, y in zip(tuple(whole) + tuple(ship), tuple(a) + tuple(b)):
        assert torch.equal(x, y)
