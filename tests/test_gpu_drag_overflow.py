"""Drag where the relative velocity, or its square, has no finite value: the
quadratic law's (v / |v|) (c A |v|^2) is then not a number, and the element is held
(jax_simulation.py:167-192, :239-254), whichever way the substeps' work is split."""
import numpy as np
import pytest
import torch

from helpers import gpu_frame_step, initial_state, to_gpu_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("active", [0.02, 1.0])
def test_water_beyond_the_range_holds_the_element(golden64, dtype, active):
    from mbd_icenav_b200 import _abi
    g, dt, K = golden64, torch.float32 if dtype == "f32" else torch.float64, 2
    o_st, o_sh = initial_state(g, "window", np.float64)
    n = len(o_st.positions)
    rng = np.random.default_rng(3)
    on = rng.permutation(n) < active * n
    big = 1e20 if dtype == "f32" else 1e200  # its square overflows
    water = [(np.inf, 0.0), (-np.inf, 0.1), (0.2, np.inf), (np.inf, -np.inf), (big, 0.0), (0.1, -big)]
    who = np.flatnonzero(on)[:len(water)]
    assert len(who) == len(water)
    vel = rng.normal(0, 0.2, (n, 2)) * on[:, None]
    st0, sh0 = to_gpu_state(o_st._replace(velocities=vel, elem_active=on), o_sh, dt)
    sp = torch.zeros((K, 6), dtype=dt, device="cuda")
    sp[:, :3], sp[:, 3:] = sh0.eta, sh0.eta
    vw = torch.zeros((K, n, 2), dtype=dt, device="cuda")
    vw[:, torch.as_tensor(who, device="cuda")] = torch.tensor(water, dtype=dt, device="cuda")
    ref = None
    for split in (_abi.DEM_SPLIT_THREAD, _abi.DEM_SPLIT_AUTO, _abi.DEM_SPLIT_WARP):
        fs = gpu_frame_step(g, "window", dt, bucket_capacity=64)
        fs.set_work_split(split, 0)
        st, sh, _ = fs.scan_segment(st0, sh0, sp, vw)
        fs.close()
        assert not st.velocities[who].any(), split
        assert torch.equal(st.positions[who], st0.positions[who]), split
        for a, b in zip(tuple(st) + tuple(sh), ref or tuple(st) + tuple(sh)):
            assert torch.equal(a, b), split
        ref = tuple(st) + tuple(sh)
